"""The row-wise kernels of portions against the ones of a few rows, which other tests hold to their formulas: where both sum in
one order the bits are the same, whatever the sizes, the column where values begin and how a row's columns fall over the threads."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# (query heads, key heads, maps, head size, value size, turned dimensions, values are the keys)
@pytest.mark.parametrize("sizes", [(6, 2, 1, 32, 40, 24, False), (5, 2, 2, 64, 128, 64, False), (3, 1, 1, 64, 4, 0, False),
                                   (4, 2, 1, 128, 128, 128, True), (1, 1, 1, 32, 32, 8, True), (64, 16, 2, 64, 128, 64, False),
                                   (70, 8, 1, 128, 128, 64, False)], ids=str)
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_query_key_norms_of_portions(sizes, dtype):
    from flambeau_b200.cache.manager import LayerCacheView
    from flambeau_b200.kernels import ops
    H, K, maps, d, e, rot, shared = sizes
    dt, page, n = getattr(torch, dtype), 8, 77
    G, cols = K // maps, (H + K) * d + (0 if shared else K // maps * e)
    g = torch.Generator(device=DEV).manual_seed(H)
    shares = torch.randn(2, n, (cols + 11) // 8 * 8, generator=g, device=DEV)
    bias = torch.randn((H + K) * d + G * e, generator=g, device=DEV).to(dt)
    qw, kw = ((torch.randn(d, generator=g, device=DEV) + 2.0).to(dt) for _ in range(2))
    table = torch.randperm(40, generator=g, device=DEV).to(torch.int32)
    positions = torch.randperm(40 * page, generator=g, device=DEV)[:n].to(torch.int32)
    angles = torch.randn(n, max(rot // 2, 1), generator=g, device=DEV)
    cos, sin = (angles.cos(), angles.sin()) if rot else (None, None)
    for norm, with_bias, parts, writable in ((True, True, 2, True), (True, False, 1, True), (False, True, 2, True), (True, False, 2, False)):
        got = []
        for step in (n, 32):                           # all rows at once; a few at a time
            cache = LayerCacheView(torch.zeros((40, G, page, maps * d), dtype=dt, device=DEV), torch.zeros((40, G, page, e), dtype=dt, device=DEV),
                                   table[None].contiguous(), i32([0]), page, writable, 0, None)
            q_out, status = torch.zeros((n, H * d), dtype=dt, device=DEV), i32([0])
            for a in range(0, n, step):
                b = min(n, a + step)
                ops.qk_norm_rope_kv_write(shares[0, a:b], qw if norm else None, kw if norm else None, "head" if norm else None, 1e-3, 0.5,
                                          cos[a:b].contiguous() if rot else None, sin[a:b].contiguous() if rot else None, rot // 2, q_out[a:b], cache,
                                          positions[a:b].contiguous(), i32([0] * (b - a)), H, K, d, e, status, n_partials=parts,
                                          partial_stride=shares.stride(0), bias=bias if with_bias else None, maps=maps,
                                          **(dict(v_off=H * d) if shared else {}))
            assert int(status) == 0
            got.append((q_out, cache.k_pool, cache.v_pool))
        for a, b in zip(*got):
            assert torch.equal(a, b)
        assert float(got[0][0].float().abs().max()) > 0


def fma(a, b, c):
    """Rounded once: a float32 product is exact in float64 (and twice-rounded sums are rare: none among these numbers)."""
    return (a.double() * b.double() + c.double()).float()


@pytest.mark.parametrize("n", [20, 77])                # (a warp a head; a CTA a row)
@pytest.mark.parametrize("d,rot", [(32, 24), (64, 64), (64, 0), (128, 128), (128, 64)])
def test_order_of_the_norm_and_the_rotation(n, d, rot):
    """Bit by bit what the sum of squares and the rotation are written as."""
    from flambeau_b200.cache.manager import LayerCacheView
    from flambeau_b200.kernels import ops
    H, half, page = 6, rot // 2, 8
    g = torch.Generator(device=DEV).manual_seed(d + n)
    proj = torch.randn(n, 2 * H * d + H * d, generator=g, device=DEV)
    weight = torch.randn(d, generator=g, device=DEV) + 2.0
    angles = torch.randn(n, max(half, 1), generator=g, device=DEV)
    cos, sin = angles.cos(), angles.sin()
    pools = [torch.zeros(10, H, page, d, device=DEV) for _ in range(2)]
    cache = LayerCacheView(*pools, i32([list(range(10))]), i32([0]), page, True, 0, None)
    for norm in (False, True):
        q, status = torch.zeros(n, H * d, device=DEV), i32([0])
        ops.qk_norm_rope_kv_write(proj, weight if norm else None, weight if norm else None, "head" if norm else None, 1e-3, 0.0,
                                  cos if rot else None, sin if rot else None, half, q, cache, i32(list(range(n))), i32([0] * n), H, H, d, d, status)
        assert int(status) == 0
        keys = pools[0].transpose(1, 2).reshape(-1, H, d)[:n]
        for got, x in ((q.view(n, H, d), proj[:, :H * d].view(n, H, d)), (keys, proj[:, H * d:2 * H * d].view(n, H, d))):
            if norm:
                v = x.reshape(n, H, d // 4, 4).unbind(-1)
                s = fma(v[3], v[3], fma(v[2], v[2], fma(v[0], v[0], v[1] * v[1])))
                while s.shape[-1] > 1:                 # lanes that differ in their highest bit meet first
                    s = s[..., :s.shape[-1] // 2] + s[..., s.shape[-1] // 2:]
                x = x * ((1.0 / torch.sqrt(s / d + 1e-3)) * weight)
            if rot:
                a, b, c, e = x[..., :half], x[..., half:rot], cos[:, None], sin[:, None]
                x = torch.cat([fma(b, -e, a * c), fma(a, e, b * c), x[..., rot:]], -1)
            assert torch.equal(got, x)


@pytest.mark.parametrize("sizes", [(2, 4, 128, 128, 4), (1, 3, 20, 36, 3), (2, 2, 136, 256, 4), (3, 3, 64, 8, 2), (2, 4, 32, 32, 1)], ids=str)
@pytest.mark.parametrize("lengths", [(77,), (3, 1, 70), (40, 9, 2, 30), (1, 1, 8, 7, 60)], ids=str)
def test_recurrences_prepared_in_portions(sizes, lengths):
    """Requests that end within a warp's rows, portions shorter than the taps, kept inputs."""
    from flambeau_b200.kernels import ops
    G, H, dk, dv, taps = sizes
    g = torch.Generator(device=DEV).manual_seed(sum(lengths))
    C = 2 * G * dk + H * dv
    cols, n, R = (C + 2 * H + 3) // 4 * 4, sum(lengths), len(lengths)
    proj = torch.randn(2, n, cols, generator=g, device=DEV)
    conv, a_log, dt_bias = (torch.randn(s, generator=g, device=DEV) for s in ((C, taps), (H,), (H,)))
    size = H * dk * dv
    state = torch.randn(R, size + max(taps - 1, 1) * C, generator=g, device=DEV)
    state = torch.nn.functional.pad(state, (0, -state.shape[1] % 4)).contiguous()
    for parts in (1, 2):
        got = []
        for alone in (False, True):                    # one step for all requests; a row at a time
            kept = state.clone()
            qkv, beta, decay = torch.zeros(n, C, device=DEV), torch.zeros(n, H, device=DEV), torch.zeros(n, H, device=DEV)

            def step(rows, slots, lens):
                a, b = rows
                starts = [sum(lens[:i]) for i in range(len(lens))]
                seq = [i for i, l in enumerate(lens) for _ in range(l)]
                batch = SimpleNamespace(row_seq=i32(seq),
                                        seq_q_start_d=i32(starts), seq_q_len_d=i32(lens), seq_slot_d=i32(slots), n_seqs=len(lens))
                ops.gdr_prepare(proj[0, a:b], conv, taps, a_log, dt_bias, kept, size, batch, qkv[a:b], beta[a:b], decay[a:b], G, H, dk, dv,
                                dk ** -0.5, 1e-6, parts, proj.stride(0))
            if alone:
                at = 0
                for s, l in enumerate(lengths):
                    for t in range(l):
                        step((at + t, at + t + 1), [s], [1])
                    at += l
            else:
                step((0, n), list(range(R)), list(lengths))
            got.append((qkv, beta, decay, kept))
        for a, b in zip(*got):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dv", [4, 36, 128, 200, 512])
@pytest.mark.parametrize("gate", [0, 1, 2])
def test_gated_norm_of_a_recurrence(dv, gate):
    from flambeau_b200.kernels import ops
    n, H = 9, 5
    g = torch.Generator(device=DEV).manual_seed(dv)
    o, proj = torch.randn(n, H * dv, generator=g, device=DEV), torch.randn(2, n, H * dv + 8, generator=g, device=DEV)
    w = torch.randn(dv, generator=g, device=DEV)
    for off in (4, 3):                                 # (columns on 16-byte borders: four channels a lane; else one)
        out = torch.zeros(n, H * dv, device=DEV)
        ops.gdr_out_norm(o, proj[0], off, w, 1e-5, out, H, dv, 2, proj.stride(0), ("silu", "sigmoid", None)[gate])
        x = o.double().view(n, H, dv)
        z = proj.double().sum(0)[:, off:off + H * dv].view(n, H, dv)
        z = [torch.nn.functional.silu(z), torch.sigmoid(z), z][gate]
        want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double() * z
        # a sum of dv squares and a handful of roundings
        assert float((out.double().view(n, H, dv) - want).abs().max()) <= (dv / 32 + 20) * 2.0 ** -24 * float(want.abs().max())
