"""The map per head of portions (tcgen05) against float64: row counts around its tiles, every size, heads with numbers between
them, shares; and what it leaves to the kernel of 64 x 64 tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 129, 255, 300, 1031])
@pytest.mark.parametrize("N,K", [(64, 64), (256, 128), (128, 256), (192, 64), (64, 512), (256, 192)])
@pytest.mark.parametrize("shares", [0, 1, 3])
def test_rows_of_heads(n, N, K, shares):
    from flambeau_b200.kernels import ops
    H, apad, opad = 3 if shares < 2 else 150, 8, 16         # (shares: where every SM has a tile)
    g = torch.Generator(device="cuda").manual_seed(n + N)
    w = torch.randn(H, N, K, generator=g, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = torch.randn(max(shares, 1), n, H * (K + apad), generator=g, device="cuda")
    a = a if shares else a.bfloat16()
    out = torch.full((n, H * (N + opad)), 7.0, device="cuda").bfloat16()
    ops.head_linear(a[0], K + apad, w, out, N + opad, n, n_partials=max(shares, 1), partial_stride=a.stride(0), status=status)
    assert int(status) == 0
    x = a.sum(0) if shares < 3 else (a[0] + a[1]) + a[2]                   # float32 shares are added in their order
    x = x.bfloat16().double().view(n, H, K + apad)[..., :K]
    want, size = (torch.einsum("nhk,hck->nhc", p, q) for p, q in ((x, w.double()), (x.abs(), w.double().abs())))
    got = out.double().view(n, H, N + opad)
    assert bool(((got[..., :N] - want).abs() <= K * 2.0 ** -23 * size + 2.0 ** -8 * want.abs() + 1e-30).all())
    assert bool((got[..., N:] == 7.0).all())


@pytest.mark.parametrize("n", [128, 300])
@pytest.mark.parametrize("N,K", [(256, 128), (128, 128), (192, 64), (256, 192), (64, 64), (128, 256)])
@pytest.mark.parametrize("H", [40, 80])                     # (float32 from half of the SMs on, and not towards fewer outputs)
def test_rows_of_many_heads(H, N, K, n):
    """One float32 share and bfloat16, on either side of the tiles from which on the kernel takes them: the same map."""
    from flambeau_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(n + N + H)
    w = torch.randn(H, N, K, generator=g, device="cuda").bfloat16()
    a, status = torch.randn(n, H * K, generator=g, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    x = a.bfloat16().double().view(n, H, K)
    want, size = (torch.einsum("nhk,hck->nhc", p, q) for p, q in ((x, w.double()), (x.abs(), w.double().abs())))
    for inputs in (a, a.bfloat16()):
        out = torch.full((n, H * N), 7.0, device="cuda").bfloat16()
        ops.head_linear(inputs, K, w, out, N, n, status=status)
        assert int(status) == 0
        assert bool(((out.double().view(n, H, N) - want).abs() <= K * 2.0 ** -23 * size + 2.0 ** -8 * want.abs() + 1e-30).all())


def test_left_to_the_other_kernel():
    """Few rows, sizes off 64, rows off 16-byte borders: the same map by the kernel of 64 x 64 tiles."""
    from flambeau_b200.kernels import ops
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for n, N, K, pad in ((127, 64, 64, 0), (200, 72, 64, 0), (200, 64, 40, 0), (200, 320, 64, 0), (200, 64, 64, 1)):
        a, w = torch.randn(n, 2 * K + pad, device="cuda").bfloat16(), torch.randn(2, N, K, device="cuda").bfloat16()
        outs = [torch.zeros(n, 2 * N, device="cuda").bfloat16() for _ in range(2)]
        ops.head_linear(a, K, w, outs[0], N, n, status=status)
        ops.head_linear(a, K, w, outs[1], N, n)
        assert torch.equal(*outs) and float(outs[0].abs().max()) > 0


@pytest.mark.parametrize("rank", [64, 128])
def test_a_portion_whose_maps_and_attention_fit_an_sm_together(rank):
    """Latents of 64 and 128: a block of the map and one of the attention behind it, which takes all of tensor memory before it
    waits, have room on an SM side by side; more of both than there are SMs."""
    from flambeau_b200.cache.manager import CallPlan
    from flambeau_b200.parts.latent_attention import LatentAttention
    from test_parts_gpu import Bench, bind_random, rel
    n, w, H, d, e = 1280, 256, 16, 128 if rank == 64 else 64, 64
    part = LatentAttention(None, "m.", width=w, num_heads=H, head_dim=d, rot_dim=0, value_dim=e, kv_rank=rank, q_rank=None,
                           window=0, scale=d ** -0.5, eps=1e-5, gate=False)
    b = Bench("bfloat16", [CallPlan(kv=part.cache_requirement())], cache_tokens=4096, max_step_tokens=n)
    part.runtime = b.rt
    W = {name[2:]: t for name, t in bind_random(part, torch.bfloat16).items()}
    ctx, _ = b.begin([("a", [1] * n, [])], w)
    h = torch.randn(n, w, generator=torch.Generator().manual_seed(rank)).bfloat16()
    part.forward(ctx, h.cuda(), ctx.delta, 0)
    b.end()
    y = ctx.delta_slabs[:ctx.pending_slabs].sum(0)
    h = h.double()
    z = h @ W["dkv"].T
    c = z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-5) * W["dkv.norm"]
    q = (h @ W["q"].T).view(n, H, d)
    uk, uv = W["uk"].view(H, d, rank), W["uv"].view(H, e, rank)
    seen = torch.ones(n, n, dtype=torch.bool).tril()
    heads = [torch.softmax((q[:, i] @ uk[i] @ c.T * d ** -0.5).masked_fill(~seen, -torch.inf), -1) @ c @ uv[i].T for i in range(H)]
    # five roundings to bfloat16 on the way (queries, latents, both maps' results, heads), of numbers no larger than the result's
    assert rel(y, torch.cat(heads, -1) @ W["o"].T) < 5 * 2.0 ** -9
