"""The recurrences over a request's tokens (csrc/recurrence.cu) against their formulas in float64, token by token: blocks of
four tokens and what is left of them, stages of shared memory and their edges, requests of different lengths in one step,
key sizes in every range of lanes (aligned rows and others), value sizes that leave columns over."""
import pytest
import torch

from test_fegizen_gpu import fake_batch

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda:0", torch.float64

LENGTHS = [[1, 1, 1], [3, 2, 1], [2, 5], [4, 1, 3], [31, 64], [33, 7, 66], [100]]
# (key size, value size, heads, query/key heads)
SIZES = [(4, 3, 2, 1), (16, 40, 2, 2), (18, 70, 2, 1), (32, 33, 4, 2), (64, 17, 2, 1), (100, 40, 2, 2), (128, 128, 4, 2), (128, 33, 20, 20),
         (128, 100, 30, 10), (127, 16, 2, 2), (200, 20, 2, 1), (256, 31, 1, 1), (500, 9, 1, 1), (600, 5, 1, 1), (1024, 6, 1, 1)]


def stepped(rule, q, k, v, beta, g, S):
    """One head and request: q, k, g [n, dk], v [n, dv], beta [n], S [dv, dk]."""
    out = []
    for t in range(q.shape[0]):
        S = S * g[t]
        u = v[t] if rule == "linear" else beta[t] * (v[t] - S @ k[t])
        S = S + u[:, None] * k[t]
        out.append(S @ q[t])
    return torch.stack(out), S


@pytest.mark.parametrize("lengths", LENGTHS, ids=str)
@pytest.mark.parametrize("sizes", SIZES, ids=str)
@pytest.mark.parametrize("rule", ["head", "channel", "linear"])
def test_recurrence_equals_its_formula(rule, sizes, lengths):
    from flambeau_b200.kernels import ops
    dk, dv, H, G = sizes
    G = H if rule == "linear" else G
    n, slots = sum(lengths), len(lengths) + 1
    gen = torch.Generator().manual_seed(dk * 7 + n)
    rand = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    q, k, v = rand(n, G, dk) * dk ** -0.5, rand(n, G, dk), rand(n, H, dv)
    k = k / k.norm(dim=-1, keepdim=True)
    beta, decay = torch.rand(n, H, generator=gen), torch.rand(n, H, dk if rule != "head" else 1, generator=gen) ** 0.25
    state = rand(slots, H * dv * dk + 8)               # (what lies behind the matrices must not be touched)
    qkv = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)], 1)
    slot_of = [slots - 1 - i for i in range(len(lengths))]
    batch = fake_batch(lengths, slot_of)
    sd, o = state.to(DEV), torch.empty(n, H * dv, device=DEV)
    qd, bd, gd = qkv.to(DEV), beta.to(DEV), decay.reshape(n, -1).contiguous().to(DEV)
    if rule == "linear":
        ops.gla_recurrent(qd, gd, sd, batch, o, H, dk, dv)
    else:
        (ops.gdr_recurrent if rule == "head" else ops.gdr_channel_recurrent)(qd, bd, gd, sd, batch, o, G, H, dk, dv)
    want_o, want_s, start = torch.empty(n, H, dv, dtype=F64), state.double(), 0
    for slot, length in zip(slot_of, lengths):
        a, b = start, start + length
        for h in range(H):
            i, at = h // (H // G), h * dv * dk
            S = want_s[slot, at:at + dv * dk].view(dv, dk)
            out, S = stepped(rule, q[a:b, i].double(), k[a:b, i].double(), v[a:b, h].double(), beta[a:b, h].double(),
                             decay[a:b, h].double().expand(length, dk), S.clone())
            want_o[a:b, h] = out
            want_s[slot, at:at + dv * dk] = S.reshape(-1)
        start = b
    # float32 sums of at most a few hundred terms that decay: a few roundings of 6e-8 each
    scale_o, scale_s = float(want_o.abs().max()), float(want_s.abs().max())
    assert float((o.double().cpu().view(n, H, dv) - want_o).abs().max()) < 4e-6 * scale_o
    assert float((sd.double().cpu() - want_s).abs().max()) < 4e-6 * scale_s


def run(rule, qkv, beta, decay, state, lengths, slots, sizes):
    from flambeau_b200.kernels import ops
    dk, dv, H, G = sizes
    batch, st, o = fake_batch(lengths, slots), state.clone(), torch.empty(sum(lengths), H * dv, device=DEV)
    batch.max_q_len = max(lengths)
    if rule == "linear":
        ops.gla_recurrent(qkv, decay, st, batch, o, H, dk, dv)
    else:
        (ops.gdr_recurrent if rule == "head" else ops.gdr_channel_recurrent)(qkv, beta, decay, st, batch, o, G, H, dk, dv)
    return o, st


@pytest.mark.parametrize("sizes", [(128, 128, 16, 4), (128, 40, 8, 8), (64, 64, 4, 2), (96, 33, 4, 4), (127, 20, 4, 4), (200, 24, 2, 2),
                                   (256, 64, 3, 3), (512, 16, 4, 4), (700, 8, 2, 2)], ids=str)
@pytest.mark.parametrize("rule", ["head", "channel", "linear"])
def test_a_request_has_the_same_bits_whatever_shares_its_step(rule, sizes):
    """Every request alone, with one other and with all others: a decoded token in a step of such tokens and beside portions,
    a portion that has the device to itself and one that shares it."""
    dk, dv, H, G = sizes
    G = H if rule == "linear" else G
    sizes = (dk, dv, H, G)
    lengths = [1, 90, 2, 343, 1, 3, 64, 7]
    gen = torch.Generator(device=DEV).manual_seed(dk + dv)
    n, starts = sum(lengths), [sum(lengths[:i]) for i in range(len(lengths))]
    qkv = torch.randn(n, 2 * G * dk + H * dv, generator=gen, device=DEV) * dk ** -0.5
    beta, decay = (torch.rand(n, w, generator=gen, device=DEV) ** 0.25 for w in (H, H * dk if rule != "head" else H))
    state = torch.randn(len(lengths), H * dv * dk, generator=gen, device=DEV)
    whole, st_whole = run(rule, qkv, beta, decay, state, lengths, list(range(len(lengths))), sizes)
    for i, length in enumerate(lengths):
        for others in ([], [0], [3], [4, 0], [2, 5]):
            who = [i] + [x for x in others if x != i]
            rows = torch.cat([torch.arange(starts[x], starts[x] + lengths[x], device=DEV) for x in who])
            o, st = run(rule, qkv[rows], beta[rows], decay[rows], state, [lengths[x] for x in who], who, sizes)
            assert torch.equal(o[:length], whole[starts[i]:starts[i] + length]), (i, who)
            assert torch.equal(st[i], st_whole[i]), (i, who)
