"""Prompt attention with two query tiles per block (csrc/kernels/attn_prefill_tc.cu), which batches of enough rows take, against
64 bits: ragged tiles, one tile of two, portions behind cached tokens, windows, kept tokens, soft caps and sinks."""
import pytest
import torch

from xllm_b200 import ops

pytestmark = pytest.mark.gpu


def _oracle(q, kc, vc, bt, cu, lens, scale, causal, window, keep, softcap, sink):
    page, out = kc.shape[2], torch.zeros(q.shape, dtype=torch.float64, device=q.device)
    for i in range(lens.shape[0]):
        b, e, n = int(cu[i]), int(cu[i + 1]), int(lens[i])
        if e == b:
            continue
        pages = bt[i, :-(-n // page)].long()
        k, v = (c[pages].transpose(1, 2).reshape(-1, c.shape[1], 128)[:n].double().repeat_interleave(q.shape[1] // c.shape[1], 1)
                for c in (kc, vc))
        s = torch.einsum("nhd,thd->hnt", q[b:e].double(), k) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        pos, t = torch.arange(n - (e - b), n, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
        seen = (t <= pos) if causal else torch.ones_like(t <= pos)
        if window:
            seen = seen & ((t > pos - window) | (t < keep))
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(-1, e - b, 1)], dim=2)
        p = torch.softmax(s, dim=2)[..., :n]
        out[b:e] = torch.einsum("hnt,thd->nhd", p, v)
    return out


def _case(lens, behind, page, nq=32, nkv=8):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + page)
    T = sum(lens)
    kv = [a + b for a, b in zip(lens, behind)]
    per = max(-(-n // page) for n in kv)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, kc, vc = rnd(T, nq, 128) * 2, rnd(len(lens) * per + 1, nkv, page, 128), rnd(len(lens) * per + 1, nkv, page, 128)
    bt = (1 + torch.randperm(len(lens) * per, device="cuda", generator=g)).view(len(lens), per).int()
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).int()
    return g, q, kc, vc, bt, cu, torch.tensor(kv, dtype=torch.int32, device="cuda")


# the last three: prompts whose mean length lies below, at and above what two tiles a block are taken from
@pytest.mark.parametrize("page", [16, 64, 128])
@pytest.mark.parametrize("options", [{}, {"window": 100}, {"window": 200, "keep": 5}, {"softcap": 3.0}, {"softcap": 50.0, "window": 300},
                                     {"causal": False}, {"sink": True}])
@pytest.mark.parametrize("lens,behind", [([700, 300, 129, 385], [0, 0, 0, 0]), ([256, 1, 257, 900], [130, 77, 0, 511]),
                                         ([100] * 9 + [300], [0, 40] * 5), ([130] * 7 + [242], [0] * 8), ([130] * 7 + [250], [0] * 8)])
def test_two_tiles(lens, behind, options, page):
    g, q, kc, vc, bt, cu, kvl = _case(lens, behind, page)
    nq = q.shape[1]
    o = {"causal": True, "window": 0, "keep": 0, "softcap": 0.0, "sink": None, **options}
    if o["sink"]:
        o["sink"] = torch.randn(nq, device="cuda", generator=g) * 2
    got = ops.paged_prefill_attention(q, kc, vc, bt, cu, kvl, max(lens), 128 ** -0.5, **o)
    want = _oracle(q, kc, vc, bt, cu, kvl, 128 ** -0.5, o["causal"], o["window"], o["keep"], o["softcap"], o["sink"])
    # weights and results are rounded to bf16, 2^-9 at most each; soft caps by a polynomial or hardware tanh add about as much
    assert (got.double() - want).norm() <= 2 ** -8 * want.norm()
    worst = (got.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert float(worst.max()) <= 2 ** -6


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens,behind", [([700, 300, 129, 385], [0, 0, 0, 0]), ([256, 1, 257, 900], [130, 77, 0, 511]),
                                         ([100] * 9 + [300], [0, 40] * 5)])
def test_log_sum_exps(lens, behind, causal):
    from xllm_b200.ops import _lib, xattn  # noqa: F401 (declares the entry point)
    from xllm_b200.ops._lib import check, ptr, stream
    _, q, kc, vc, bt, cu, kvl = _case(lens, behind, 16)
    T, nq, nkv, out = q.shape[0], q.shape[1], kc.shape[1], torch.empty_like(q)
    lse = torch.full((T, nq), 7.0, device="cuda")
    check(_lib.load().xllm_paged_prefill_attn_tc_lse(ptr(out), out.stride(0), ptr(q), q.stride(0), T, ptr(kc), ptr(vc), kc.shape[0],
                                                     ptr(bt), bt.stride(0), ptr(cu), ptr(kvl), len(lens), max(lens), nq, nkv, 16,
                                                     128 ** -0.5, int(causal), 0, ptr(lse), stream()), "lse")
    for i, n in enumerate(kvl.tolist()):
        b, e = int(cu[i]), int(cu[i + 1])
        k = kc[bt[i, :-(-n // 16)].long()].transpose(1, 2).reshape(-1, nkv, 128)[:n].double().repeat_interleave(nq // nkv, 1)
        s = torch.einsum("nhd,thd->hnt", q[b:e].double(), k) * 128 ** -0.5
        if causal:
            pos = torch.arange(n - (e - b), n, device="cuda")[:, None]
            s = s.masked_fill(torch.arange(n, device="cuda")[None] > pos, float("-inf"))
        want = torch.logsumexp(s, dim=2).T * 1.4426950408889634
        # scores in fp32 and exponentials of 2^-22: sums of up to 1400 positive terms
        assert float((lse[b:e].double() - want).abs().max()) <= 1e-4
