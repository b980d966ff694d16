"""Portions of prompts on the tcgen05 attention kernel with softmax weights of two or three bfloat16 numbers each, and over cache rows
that are keys and values at once, against a softmax in float64: heads of 64, 128 and 256, one to 64 query heads a key/value
head, portions around the edges of row tiles and key tiles, decoded tokens whose keys are cut into stretches, windows that
cut a page, pages of 8 to 64 keys, sinks, poison in every slot that was not written; on the tcgen05 kernel and with it
switched off."""
import pytest
import torch

from test_attention_gpu import Scene, prompt_kernel  # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu

# (query heads, key/value heads, head size, values are the keys)
GEOMETRY = [(32, 1, 256, True), (3, 1, 256, True), (8, 2, 256, True), (64, 1, 256, True), (8, 2, 128, False), (4, 4, 64, False), (20, 2, 128, False)]
SEQS = [[(0, 129), (37, 70)], [(100, 333)], [(5, 64), (200, 1), (63, 65)], [(1500, 1), (64, 1), (0, 1), (319, 1), (62, 2)], [(127, 1)] * 60]


def softmax_over_pages(sc, sinks, scale):
    out, dev, G = [], "cuda", sc.nh // sc.nkv
    for s, (cached, new) in enumerate(sc.seqs):
        k, v, q = (t[s].double().to(dev) for t in (sc.k, sc.v, sc.q))
        p, j = torch.arange(cached, cached + new, device=dev)[:, None], torch.arange(cached + new, device=dev)[None]
        seen = (j <= p) & ((p - j < sc.window) if sc.window else (j >= 0))
        o = torch.empty(new, sc.nh, sc.hd, dtype=torch.float64, device=dev)
        for h in range(sc.nh):
            z = ((q[:, h] @ k[:, h // G].T) * scale).masked_fill(~seen, float("-inf"))
            if sinks is not None:
                z = torch.cat([z, sinks[h].double().to(dev).expand(new, 1)], 1)
            o[:, h] = torch.softmax(z, -1)[:, :cached + new] @ v[:, h // G]
        out.append(o.reshape(new, -1))
    return torch.cat(out).cpu()


def attend(sc, sinks, scale, shared):
    """The kernel's result for a scene whose values are its keys (shared) or their own."""
    from flambeau_b200.kernels import ops
    dev, seqs = "cuda", sc.seqs
    q, kp = sc.q_flat.to(dev, torch.bfloat16), sc.k_pool.to(dev, torch.bfloat16)
    vp = kp if shared else sc.v_pool.to(dev, torch.bfloat16)
    out, status = torch.full_like(q, float("nan")), torch.zeros(1, dtype=torch.int32, device=dev)
    multi = [s for s, (_, n) in enumerate(seqs) if n > 1]
    short = [ops.attention_is_short(n, sc.nh, sc.nkv) for _, n in seqs]
    ops.paged_attention_mma(q, out, kp, vp, sc.table.to(dev), sc.seq_q_start.to(dev), sc.seq_q_len.to(dev), sc.seq_pos_start.to(dev),
                            len(seqs), max(n for _, n in seqs), max(c + n for c, n in seqs), any(short), not all(short), sc.nh, sc.nkv,
                            sc.hd, sc.window, scale, status, table_base=sc.table_base.to(dev), n_multi=len(multi),
                            multi_seqs=torch.tensor(multi + [0], dtype=torch.int32, device=dev), sinks=sinks.to(dev),
                            weights_float32=True)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return out


@pytest.mark.parametrize("seqs", SEQS, ids=str)
@pytest.mark.parametrize("window,page", [(0, 16), (50, 16), (0, 8), (97, 64)])
@pytest.mark.parametrize("geometry", GEOMETRY, ids=str)
def test_portions_with_weights_in_two_parts(prompt_kernel, geometry, window, page, seqs):
    nh, nkv, hd, shared = geometry
    sc = Scene(seqs, nh, nkv, hd, window, torch.bfloat16, page_size=page, seed=hd + window, compact=True)
    if shared:
        sc.v, sc.v_pool = sc.k, sc.k_pool
    sinks, scale = torch.randn(nh), hd ** -0.5
    out = attend(sc, sinks, scale, shared)
    want = softmax_over_pages(sc, sinks, scale)
    assert bool(torch.isfinite(out).all()), "poison from a slot that was not written"
    # one rounding of the result (half a unit in the last of 8 bits: at most 2^-8 of a value), and the weights' own remainder
    # (2^-17 of a weight, weighing values of the largest size)
    err, most = (out.double().cpu() - want).abs(), float(want.abs().max())
    assert bool((err <= 2.0 ** -8 * want.abs() + 2.0 ** -14 * most).all())


@pytest.mark.parametrize("geometry,seqs", [((32, 1, 256, True), [(1000, 300)]), ((32, 1, 256, True), [(200, 1)] * 64),
                                           ((8, 2, 128, False), [(500, 700)]), ((8, 2, 128, False), [(100, 40)]),
                                           ((32, 4, 128, False), [(0, 1500)]), ((8, 2, 64, False), [(500, 700)])],
                         ids=lambda x: str(x) if len(x) < 9 else "decoded")
def test_weights_lose_no_more_than_on_the_mma_sync_kernel(geometry, seqs):
    """Uneven weights: how many results are not the rounding of the exact ones.  Every weight's own error makes some results
    cross a border between two bfloat16 numbers; the largest weight of a row, which counts most, has none where it is 1."""
    from flambeau_b200.kernels import ops
    nh, nkv, hd, shared = geometry
    sc = Scene(seqs, nh, nkv, hd, 0, torch.bfloat16, seed=hd + len(seqs), compact=True, spread=3.0 ** 0.5)
    if shared:
        sc.v, sc.v_pool = sc.k, sc.k_pool
    sinks, scale, wrong = torch.randn(nh), hd ** -0.5, []
    want = softmax_over_pages(sc, sinks, scale).float().bfloat16()
    for on in (True, False):
        ops.set_attention_tc(on)
        try:
            wrong.append(int((attend(sc, sinks, scale, shared).cpu() != want).sum()))
        finally:
            ops.set_attention_tc(True)
    # (counts of rare events: three standard deviations of their difference)
    assert wrong[0] <= wrong[1] + 3.0 * sum(wrong) ** 0.5, wrong
