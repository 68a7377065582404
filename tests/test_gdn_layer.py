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
# (decode rows, prompt lengths): tiles of 16 tokens and runs of 4 rows met exactly, missed by one, and long prompts; prompts without
# rows, as the captured steps have them
BATCHES = [(1, []), (5, []), (0, [1, 16, 17, 2]), (3, [3, 15, 33, 130]), (2, [0, 20, 0, 0])]


class Batch:
    """Inputs and states of a layer, and what `run` makes of them on the GPU."""

    def __init__(self, nk, nv, dk, dv, taps, packed, decode, prompts, go_on=True):
        g = self.g = torch.Generator().manual_seed(nk * 1000 + dk + dv + taps + decode + sum(prompts))
        self.dk, self.dv, self.packed, self.decode = dk, dv, packed, decode
        n_seqs, pad = decode + len(prompts), 2 if prompts else 0          # rows behind the last sequence
        self.cu = torch.tensor([0] + [1] * decode + prompts).cumsum(0).int()
        T = self.T = int(self.cu[-1]) + pad
        self.slots = torch.randperm(n_seqs + 2, generator=g)[:n_seqs].int()
        self.lens = (self.cu[1:] - self.cu[:-1]).clone()
        if go_on:
            self.lens[::2] += 40                                          # every other sequence goes on
        if n_seqs > 3:
            self.slots[2] = -1                                            # and one row or portion is padding
        rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).to(torch.bfloat16)
        self.x = {"q": rnd(T, nk, dk), "k": rnd(T, nk, dk), "v": rnd(T, nv, dv), "z": rnd(T, nv, dv), "b": rnd(T, nv), "a": rnd(T, nv)}
        C = 2 * nk * dk + nv * dv
        self.rec, self.tail = torch.randn(n_seqs + 2, nv, dk, dv, generator=g), rnd(n_seqs + 2, C, taps - 1)
        # decays from nothing forgotten to everything within a few tokens
        self.layer = gdn.GatedDelta(nk, nv, dk, dv, taps, 1e-6, rnd(C, taps, std=0.5), rnd(nv), torch.linspace(-6, 4, nv).to(torch.bfloat16),
                                    (1 + 0.1 * torch.randn(dv, generator=g)).to(torch.bfloat16))

    def live(self):
        rows = torch.zeros(self.T, dtype=torch.bool)
        for i, s in enumerate(self.slots.tolist()):
            rows[int(self.cu[i]):int(self.cu[i + 1])] = s >= 0
        return rows

    def settle(self):
        """Other inputs wherever the convolution's output lies so near the middle between two bf16 values (an eighth of a
        percent of their distance: some thirty times what fp32 sums and exponentials are off by) that it could round to either."""
        nk, nv, K = self.layer.nk, self.layer.nv, self.layer.taps
        w = self.layer.conv_w.double()
        for _ in range(100):
            left = 0
            for i, slot in enumerate(self.slots.tolist()):
                b0, b1 = int(self.cu[i]), int(self.cu[i + 1])
                n = b1 - b0
                if slot < 0 or n == 0:
                    continue
                parts = [self.x[p][b0:b1].reshape(n, -1) for p in ("q", "k", "v")]
                old = torch.zeros_like(self.tail[slot]) if int(self.lens[i]) == n else self.tail[slot]
                full = torch.cat([old.T, torch.cat(parts, dim=1)]).double()
                y = sum(full[j:j + n] * w[:, j] for j in range(K))
                y = y * torch.sigmoid(y)
                m = torch.frexp(y)[0].abs() * 256                          # bf16 holds eight bits of it
                near = ((m - m.floor() - 0.5).abs() < 1.25e-3) | (y.abs() < 1e-30)
                left += int(near.sum())
                fresh = torch.randn(near.shape, generator=self.g).to(torch.bfloat16)
                for part, bad, new in zip(("q", "k", "v"), near.split([p.shape[1] for p in parts], 1), fresh.split([p.shape[1] for p in parts], 1)):
                    here = self.x[part][b0:b1].reshape(n, -1)
                    self.x[part][b0:b1] = torch.where(bad, new, here).view(self.x[part][b0:b1].shape)
            if left == 0:
                return self
        raise AssertionError("inputs do not settle")

    def oracle(self):
        return _oracle(self.x, self.layer, self.rec, self.tail, self.slots, self.cu, self.lens, self.dk, self.dv)

    def run(self, max_q_len=None):
        """(rows, states, tails)"""
        layer, x, T, dk, dv, dev = self.layer, self.x, self.T, self.dk, self.dv, "cuda"
        nk, r = layer.nk, layer.nv // layer.nk
        grouped = lambda t: t.reshape(T, nk, -1)
        if self.packed:
            y = torch.cat([grouped(x["q"]), grouped(x["k"]), grouped(x["v"]), grouped(x["z"])], dim=2).reshape(T, -1).to(dev)
            ba = torch.cat([grouped(x["b"]), grouped(x["a"])], dim=2).reshape(T, -1).to(dev)
            width = 2 * dk + 2 * r * dv
            parts = (y, y[:, dk:], y[:, 2 * dk:], y[:, 2 * dk + r * dv:], ba, ba[:, r:], width, width, width, 2 * r)
        else:
            y = torch.cat([x["q"].reshape(T, -1), x["k"].reshape(T, -1), x["v"].reshape(T, -1)], dim=1).to(dev)
            parts = (y, y[:, nk * dk:], y[:, 2 * nk * dk:], x["z"].reshape(T, -1).to(dev), x["b"].to(dev), x["a"].to(dev), dk, r * dv,
                     r * dv, r)
        on_gpu = gdn.GatedDelta(layer.nk, layer.nv, dk, dv, layer.taps, layer.eps, *(t.to(dev) for t in (
            layer.conv_w, layer.dt_bias, layer.a_log, layer.norm_w)))
        rec, tail = self.rec.to(dev), self.tail.to(dev)
        rows = on_gpu(rec, tail, self.slots.to(dev), self.cu.to(dev), self.lens.to(dev), self.decode, *parts, max_q_len=max_q_len)
        return rows.cpu(), rec.cpu(), tail.cpu()


def _compare(batch, got, rel=1e-5):
    rows, rec, tail = got
    want_rows, want_rec, want_tail = batch.oracle()
    assert torch.equal(tail, want_tail)
    live = batch.live()
    assert not rows[~live].any()
    # fp32 sums of a few hundred terms, and a term of 2^-24 for every token that is remembered: by state and head
    off = (rec.double() - want_rec).flatten(2).norm(dim=2) / want_rec.flatten(2).norm(dim=2)
    assert float(off.max()) <= rel, float(off.max())
    # three roundings to bf16 of 2^-9 at most each
    assert (rows[live].double() - want_rows[live]).norm() <= 3 * 2 ** -9 * want_rows[live].norm()


@pytest.mark.gpu
@pytest.mark.parametrize("decode,prompts", BATCHES)
@pytest.mark.parametrize("nk,nv,dk,dv,taps,packed", SIZES)
def test_layer_matches_64_bits(nk, nv, dk, dv, taps, packed, decode, prompts):
    batch = Batch(nk, nv, dk, dv, taps, packed, decode, prompts).settle()
    _compare(batch, batch.run())
    if prompts:                                                       # as captured for longer ones
        for a, b in zip(batch.run(max_q_len=batch.T - 1), batch.run(max_q_len=max(prompts))):
            assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("go_on", [False, True])
def test_long_prompts_match_64_bits(go_on):
    batch = Batch(2, 4, 128, 128, 4, True, 0, [1030, 700], go_on).settle()
    _compare(batch, batch.run())


@pytest.mark.gpu
def test_small_decays_behind_large_ones():
    """Within a chunk, tokens that forget a thousandth behind one that forgets everything: the difference of the sums of their logs
    needs more bits than fp32 sums have (2^-15 of the decay at a sum of 1000)."""
    batch = Batch(1, 2, 64, 64, 4, False, 0, [48, 33]).settle()
    batch.layer.a_log[:] = 0.0
    batch.layer.dt_bias[:] = 0.0
    batch.x["a"][:] = -7.0
    batch.x["a"][5::16] = 1000.0
    batch.x["a"][28::31] = 4000.0
    _compare(batch, batch.run(), rel=2e-6)


# (what, row of the first prompt): inside a chunk, at its first and its last token
BAD = [(w, t) for w in ("q", "k", "v", "b", "forget") for t in (20, 32, 31)] + [("tail", 0), ("state", 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("what,at", BAD)
@pytest.mark.parametrize("nk,nv,dk,dv,taps", [(2, 4, 128, 128, 4), (1, 2, 20, 36, 3), (1, 2, 36, 100, 2)])
def test_values_that_are_not_finite_stay_behind_their_token(nk, nv, dk, dv, taps, what, at):
    """They reach later tokens of their sequence and head, as token by token, and nothing else; and a decay to zero within one token
    is none of them."""
    batch = Batch(nk, nv, dk, dv, taps, True, 1, [40, 33]).settle()      # the first and the last go on, the 40 rows begin
    if what in ("tail", "state"):
        batch.lens[1] += 3                                               # now they go on as well
        batch.settle()
    row, slot = int(batch.cu[1]) + at, int(batch.slots[1])
    if what == "q":
        batch.x["q"][row, 0, 5] = float("inf")
    elif what == "k":
        batch.x["k"][row, 0, 5] = float("nan")
    elif what == "v":
        batch.x["v"][row, 1, 3] = float("nan")
    elif what == "b":
        batch.x["b"][row, 1] = float("nan")
    elif what == "forget":
        batch.x["a"][row, 1] = float("inf")
    elif what == "tail":
        batch.tail[slot, 5, 0] = float("nan")                            # the oldest input of a query channel
    else:
        batch.rec[slot, 1, :, 7] = float("inf")
    rows, rec, tail = batch.run()
    want_rows, want_rec, want_tail = batch.oracle()
    assert bool(want_rows.isfinite().all()) == (what == "forget")
    for got, want in ((rows, want_rows), (rec, want_rec), (tail, want_tail)):
        assert torch.equal(got.isfinite(), want.isfinite())
    live, fine = batch.live(), want_rows.isfinite()
    a, b = rows[live].double()[fine[live]], want_rows[live][fine[live]]
    assert (a - b).norm() <= 3 * 2 ** -9 * b.norm()
    fine = want_rec.isfinite()
    assert (rec.double()[fine] - want_rec[fine]).norm() <= 1e-5 * want_rec[fine].norm()


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


# whole heads in halves, of every width that has a kernel of its own, and a part of a head; heads that fill no warp, a part of a
# second one, and several
@pytest.mark.gpu
@pytest.mark.parametrize("d,rot", [(64, 64), (128, 128), (256, 256), (128, 32)])
@pytest.mark.parametrize("nq,nkv", [(1, 1), (6, 2), (29, 3)])
def test_rope_reads_queries_beside_their_gates(d, rot, nq, nkv):
    from xllm_b200 import ops
    from xllm_b200.ops import reference
    g = torch.Generator().manual_seed(d + rot + nq)
    T, page, pages = 23, 16, 4
    qkv = torch.randn(T, nq * 2 * d + 2 * nkv * d, generator=g).bfloat16().cuda()
    # weights w + 1 that bf16 holds exactly: both ways add in fp32
    w = [((1 + (0.1 * torch.randn(d, generator=g)).bfloat16().cuda()) - 1) for _ in range(2)]
    cs = reference.build_cos_sin_cache(rot, 64, 1e4, None, "cuda")
    pos = torch.randint(0, 64, (T,), generator=g).cuda()
    slots = torch.randperm(pages * page, generator=g)[:T].int().cuda()
    slots[[3, T - 1]] = -1
    packed = torch.cat([qkv[:, :nq * 2 * d].view(T, nq, 2 * d)[..., :d].reshape(T, nq * d), qkv[:, nq * 2 * d:]], dim=1)
    outs = []
    for rows, extra in ((packed, dict(q_norm_w=w[0] + 1, k_norm_w=w[1] + 1)),
                        (qkv, dict(q_norm_w=w[0], k_norm_w=w[1], q_head_stride=2 * d, norm_offset=1.0))):
        caches = [torch.full((pages, nkv, page, d), 7.0, device="cuda").bfloat16() for _ in range(2)]
        outs.append([*ops.rope_kv_write(rows, nq, nkv, d, pos, cs, rot, slots=slots, k_cache=caches[0], v_cache=caches[1], eps=1e-6,
                                        return_kv=True, **extra), *caches])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    q, k, v, k_cache, v_cache = outs[1]
    for got, want in zip((q, k, v), reference.rope_kv(packed.double(), nq, nkv, d, pos, cs.double(), rot, (w[0] + 1).double(),
                                                      (w[1] + 1).double(), 1e-6, False)):
        # the normed value, and the result of two products, are rounded to bf16: 2^-9 at most each
        assert (got.double() - want).norm() <= 2 ** -8 * want.norm()
    for cache, dense in ((k_cache, k), (v_cache, v)):
        at = torch.full_like(cache, 7.0)
        for t, s in enumerate(slots.tolist()):
            if s >= 0:
                at[s // page, :, s % page] = dense[t]
        assert torch.equal(cache, at)
