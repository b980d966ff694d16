"""The counting sort of many (token, choice) pairs by warps: whatever the experts' loads (none, one that takes all, ragged),
every pair has a place of its own in a tile of its expert, pairs without an expert have none, and tiles come expert by expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,E,tile", [(512, 2, 8, 16), (1000, 6, 64, 128), (700, 3, 256, 64), (2048, 6, 64, 128), (1025, 1, 33, 16), (600, 2, 300, 16)], ids=str)
@pytest.mark.parametrize("load", ["even", "one", "ragged", "beyond"])
def test_every_pair_has_its_place(n, K, E, tile, load):
    from flambeau_b200.kernels import ops
    g = torch.Generator().manual_seed(n + E)
    chosen = torch.rand(n, E + (2 if load == "beyond" else 0), generator=g).topk(K, -1).indices.int()
    if load == "one":
        chosen[:] = E - 1
    if load == "ragged":
        chosen = torch.where(torch.rand(n, K, generator=g) < 0.7, torch.zeros_like(chosen), chosen)
    pairs, tiles = n * K, ops.moe_max_tiles(n * K, E, tile)
    i32 = dict(dtype=torch.int32, device="cuda")
    token, place, expert, pair = (torch.full((m,), -7, **i32) for m in (tiles * tile, pairs, tiles, tiles * tile))
    ops.moe_sort(chosen.cuda(), E, tile, token, place, expert, pair)
    token, place, expert, pair = (t.cpu() for t in (token, place, expert, pair))
    flat = chosen.reshape(-1)
    has = flat < E
    assert bool((place[~has] == -1).all()) and place[has].unique().numel() == int(has.sum())
    at = place[has].long()
    assert torch.equal(expert[at // tile], flat[has]) and torch.equal(token[at], (torch.arange(pairs) // K).int()[has])
    assert torch.equal(pair[at], torch.arange(pairs).int()[has]) and int((token >= 0).sum()) == int(has.sum())
    count = torch.bincount(flat[has].long(), minlength=E)
    want = torch.repeat_interleave(torch.arange(E), -(-count // tile)).int()
    assert torch.equal(expert[:want.numel()], want) and bool((expert[want.numel():] == -1).all())
