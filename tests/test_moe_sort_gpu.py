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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=str)
@pytest.mark.parametrize("width", [64, 2048, 100])
@pytest.mark.parametrize("shared", [False, True])
def test_rows_of_tiles_that_have_a_group(dtype, width, shared):
    """Fetched rows of used tiles, with and without shares and places without a token; a skipped tile keeps what it held in the
    form that moves eight numbers at a time (100 is no multiple: one number at a time writes it).  Tables that do not reach over
    all rows are refused before anything is launched."""
    from flambeau_b200.kernels import ops
    from flambeau_b200.kernels.library import KernelError
    g = torch.Generator().manual_seed(width)
    n, tile, tiles = 40, 16, 5
    rows = tiles * tile
    h = torch.randn(n, width, generator=g).to("cuda", dtype)
    token = torch.randint(0, n, (rows,), generator=g).int()
    token[torch.rand(rows, generator=g) < 0.2] = -1
    group = torch.tensor([3, -1, 0, 3, -1], dtype=torch.int32)
    share, pair = torch.rand(2 * n, generator=g), torch.randint(0, 2 * n, (rows,), generator=g).int()
    more = dict(share=share.cuda(), place_pair=pair.cuda()) if shared else {}
    out = torch.full((rows, width), 7.0, dtype=dtype, device="cuda")
    ops.gather_rows(h, token.cuda(), out, tile_group=group.cuda(), tile=tile, **more)
    want = torch.where(token[:, None] >= 0, h.cpu().float()[token.clamp_min(0).long()] * (share[pair.long()][:, None] if shared else 1.0), 0.0)
    used = (group >= 0).repeat_interleave(tile)
    assert torch.equal(out.cpu()[used], want.to(dtype)[used])
    if width % 8 == 0:
        assert bool((out.cpu()[~used] == 7.0).all())
    for bad in (dict(tile_group=group[:4].cuda(), tile=tile), dict(tile_group=group.cuda(), tile=0), dict(tile_group=group.cuda(), tile=15)):
        with pytest.raises(KernelError):
            ops.gather_rows(h, token.cuda(), out, **bad)


@pytest.mark.parametrize("rows", [192, 8256])                      # (a CTA a row; two)
def test_places_of_tiles_without_a_group_are_not_followed(rows):
    """Whatever stands there: no such token, no such pair."""
    from flambeau_b200.kernels import ops
    tile, D, tokens = 32, 136, 50
    g = torch.Generator().manual_seed(rows)
    group = torch.arange(rows // tile, dtype=torch.int32) % 3 - 1       # every third tile has none
    token, pair = (torch.randint(0, tokens, (rows,), generator=g, dtype=torch.int32) for _ in range(2))
    none = (group < 0).repeat_interleave(tile)
    token[none], pair[none] = 2 ** 31 - 1, -2 ** 31
    h, share = torch.randn(tokens, D, generator=g).bfloat16(), torch.rand(tokens, generator=g)
    for more in ({}, dict(share=share.cuda(), place_pair=pair.cuda())):
        out = torch.full((rows, D), 7.0, device="cuda").bfloat16()
        ops.gather_rows(h.cuda(), token.cuda(), out, tile_group=group.cuda(), tile=tile, **more)
        want = torch.full((rows, D), 7.0).bfloat16()
        want[~none] = h[token[~none].long()]
        if more:
            want[~none] = (want[~none].float() * share[pair[~none].long(), None]).bfloat16()
        assert torch.equal(out.cpu(), want)
