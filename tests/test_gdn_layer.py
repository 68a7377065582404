"""A gated delta net layer between its projections (ops/gdn.GatedDelta) against the same steps in 64 bits, over batches that
mix decode rows, prompt portions, padding rows and sequences that start afresh or go on."""
import pytest
import torch

from xllm_b200.ops import gdn


def _oracle(x, layer, rec, tail, slots, cu, lens, dk, dv):
    """x: dict of q, k [T, nk, dk], v, z [T, nv, dv], b, a [T, nv].  Returns (rows, rec, tail); roundings to bf16 are where the
    layer has them, everything else in 64 bits."""
    d, bf = torch.float64, torch.bfloat16
    nk, nv, K, r = layer.nk, layer.nv, layer.taps, layer.nv // layer.nk
    T = x["q"].shape[0]
    rec, tail = rec.to(d).clone(), tail.clone()
    mixed = torch.cat([x["q"].reshape(T, -1), x["k"].reshape(T, -1), x["v"].reshape(T, -1)], dim=1)
    w = layer.conv_w.to(d)
    out = torch.zeros(T, nv, dv, dtype=d)
    for i, slot in enumerate(slots.tolist()):
        b0, b1, n = int(cu[i]), int(cu[i + 1]), int(cu[i + 1] - cu[i])
        if slot < 0 or n == 0:
            continue
        fresh = int(lens[i]) == n
        S = torch.zeros_like(rec[slot]) if fresh else rec[slot].clone()
        old = torch.zeros_like(tail[slot]) if fresh else tail[slot]
        full = torch.cat([old.T, mixed[b0:b1]])
        tail[slot] = full[-(K - 1):].T
        y = sum(full[j:j + n].to(d) * w[:, j] for j in range(K))
        y = (y * torch.sigmoid(y)).to(bf).to(d)
        q, k, v = y.split([nk * dk, nk * dk, nv * dv], dim=1)
        unit = lambda t: t / (t.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        q = (unit(q.view(n, nk, dk)) * dk ** -0.5).repeat_interleave(r, 1)
        k, v = unit(k.view(n, nk, dk)).repeat_interleave(r, 1), v.view(n, nv, dv)
        beta = torch.sigmoid(x["b"][b0:b1].to(d))
        g = torch.exp(-layer.a_log.to(d).exp() * torch.nn.functional.softplus(x["a"][b0:b1].to(d) + layer.dt_bias.to(d)))
        for t in range(n):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[b0 + t] = torch.einsum("hkv,hk->hv", S, q[t])
        rec[slot] = S
    z = x["z"].to(d)
    norm = (out * torch.rsqrt(out.pow(2).mean(-1, keepdim=True) + layer.eps)).to(bf)
    rows = (layer.norm_w * norm).to(d) * (z * torch.sigmoid(z))
    return rows.reshape(T, nv * dv), rec, tail


# (key heads, value heads, dk, dv, taps, packed): whole and part warps of columns and rows, one to four taps of history
SIZES = [(2, 4, 128, 128, 4, True), (2, 2, 64, 128, 4, False), (1, 3, 32, 64, 3, True), (2, 4, 20, 36, 2, False),
         (1, 1, 100, 4, 4, True), (1, 2, 4, 100, 3, False)]
# (decode rows, prompt lengths): tiles of 16 tokens and runs of 4 rows met exactly, missed by one, and long prompts
BATCHES = [(1, []), (5, []), (0, [1, 16, 17, 2]), (3, [3, 15, 33, 130])]


@pytest.mark.gpu
@pytest.mark.parametrize("decode,prompts", BATCHES)
@pytest.mark.parametrize("nk,nv,dk,dv,taps,packed", SIZES)
def test_layer_matches_64_bits(nk, nv, dk, dv, taps, packed, decode, prompts):
    g = torch.Generator().manual_seed(nk * 1000 + dk + dv + taps + decode + sum(prompts))
    bf, r = torch.bfloat16, nv // nk
    n_seqs, pad = decode + len(prompts), 2 if prompts else 0          # rows behind the last sequence
    cu = torch.tensor([0] + [1] * decode + prompts).cumsum(0).int()
    T = int(cu[-1]) + pad
    slots = torch.randperm(n_seqs + 2, generator=g)[:n_seqs].int()
    lens = (cu[1:] - cu[:-1]).clone()
    lens[::2] += 40                                                   # every other sequence goes on
    if n_seqs > 3:
        slots[2] = -1                                                 # and one row or portion is padding
    rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).to(bf)
    x = {"q": rnd(T, nk, dk), "k": rnd(T, nk, dk), "v": rnd(T, nv, dv), "z": rnd(T, nv, dv), "b": rnd(T, nv), "a": rnd(T, nv)}
    C = 2 * nk * dk + nv * dv
    rec, tail = torch.randn(n_seqs + 2, nv, dk, dv, generator=g), rnd(n_seqs + 2, C, taps - 1)
    # decays from nothing forgotten to everything within a few tokens
    layer = gdn.GatedDelta(nk, nv, dk, dv, taps, 1e-6, rnd(C, taps, std=0.5), rnd(nv), torch.linspace(-6, 4, nv).to(bf),
                           (1 + 0.1 * torch.randn(dv, generator=g)).to(bf))
    rows, want_rec, want_tail = _oracle(x, layer, rec, tail, slots, cu, lens, dk, dv)

    dev = "cuda"
    grouped = lambda t: t.reshape(T, nk, -1)
    if packed:
        y = torch.cat([grouped(x["q"]), grouped(x["k"]), grouped(x["v"]), grouped(x["z"])], dim=2).reshape(T, -1).to(dev)
        ba = torch.cat([grouped(x["b"]), grouped(x["a"])], dim=2).reshape(T, -1).to(dev)
        width = 2 * dk + 2 * r * dv
        parts = (y, y[:, dk:], y[:, 2 * dk:], y[:, 2 * dk + r * dv:], ba, ba[:, r:], width, width, width, 2 * r)
    else:
        y = torch.cat([x["q"].reshape(T, -1), x["k"].reshape(T, -1), x["v"].reshape(T, -1)], dim=1).to(dev)
        parts = (y, y[:, nk * dk:], y[:, 2 * nk * dk:], x["z"].reshape(T, -1).to(dev), x["b"].to(dev), x["a"].to(dev), dk, r * dv,
                 r * dv, r)
    for f in ("conv_w", "dt_bias", "a_log", "norm_w"):
        setattr(layer, f, getattr(layer, f).to(dev))
    rec_d, tail_d = rec.to(dev), tail.to(dev)
    got = layer(rec_d, tail_d, slots.to(dev), cu.to(dev), lens.to(dev), decode, *parts).cpu()
    assert torch.equal(tail_d.cpu(), want_tail)
    live = torch.zeros(T, dtype=torch.bool)
    for i, s in enumerate(slots.tolist()):
        live[int(cu[i]):int(cu[i + 1])] = s >= 0
    assert not got[~live].any()
    # fp32 sums of up to a few hundred terms (1e-6), and now and then a convolution output that rounds to the other bf16
    assert (rec_d.cpu().double() - want_rec).norm() <= 1e-3 * want_rec.norm()
    # three roundings to bf16 of 2^-9 at most each
    assert (got[live].double() - rows[live]).norm() <= 3 * 2 ** -9 * rows[live].norm()


@pytest.mark.gpu
@pytest.mark.parametrize("T,heads,d", [(1, 1, 8), (3, 5, 64), (130, 16, 128)])
def test_sigmoid_gate(T, heads, d):
    g = torch.Generator().manual_seed(T)
    rows = torch.randn(T, heads * 2 * d + 24, generator=g).bfloat16()
    out = torch.randn(T, heads, d, generator=g).bfloat16()
    gate = rows[:, :heads * 2 * d].view(T, heads, 2 * d)[..., d:].double()
    want = out.double() * torch.sigmoid(gate)
    got = gdn.sigmoid_gate_(out.cuda(), rows.cuda()[:, d:], 2 * d).cpu().double()
    assert ((got - want).abs() <= 2 ** -7 * want.abs() + 1e-30).all()          # two roundings to bf16


@pytest.mark.gpu
def test_rope_reads_queries_beside_their_gates():
    from xllm_b200 import ops
    from xllm_b200.ops import reference
    g = torch.Generator().manual_seed(0)
    T, nq, nkv, d, rot = 7, 6, 2, 128, 32
    qkv = torch.randn(T, nq * 2 * d + 2 * nkv * d, generator=g).bfloat16().cuda()
    w = [(0.1 * torch.randn(d, generator=g)).bfloat16().cuda() for _ in range(2)]
    cs = reference.build_cos_sin_cache(rot, 64, 1e4, None, "cuda")
    pos = torch.arange(T).cuda()
    packed = torch.cat([qkv[:, :nq * 2 * d].view(T, nq, 2 * d)[..., :d].reshape(T, nq * d), qkv[:, nq * 2 * d:]], dim=1)
    # weights w + 1 that bf16 holds exactly: both ways add in fp32
    w = [((1 + x) - 1) for x in w]
    kw = dict(eps=1e-6, return_kv=True)
    want = ops.rope_kv_write(packed, nq, nkv, d, pos, cs, rot, q_norm_w=w[0] + 1, k_norm_w=w[1] + 1, **kw)
    got = ops.rope_kv_write(qkv, nq, nkv, d, pos, cs, rot, q_norm_w=w[0], k_norm_w=w[1], q_head_stride=2 * d, norm_offset=1.0, **kw)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
