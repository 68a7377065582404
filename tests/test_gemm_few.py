"""Products of few rows (csrc/kernels/gemm_few.cu): bf16 with bias or gated activation, block-scaled fp8, and both grouped by
expert, against 64 bits."""
import pytest
import torch

from xllm_b200.ops import fp8, gemm_tcgen05, glu, moe

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, want, rel):
    assert (got.double() - want).norm() <= rel * want.norm(), float((got.double() - want).norm() / want.norm())


# column tiles of 16, 32 and 64 met and missed by one; weight rows below, at and behind a tile of 128; K below a block, with
# a tail, one slice and several (the fewer tiles of weights, the more slices), and more tiles than SMs
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 8), (64, 200), (128, 64), (576, 7168), (1544, 4096), (20000, 256)])
def test_bf16(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    x = torch.randn(M, K + 8, device=DEV, generator=g).bfloat16()[:, :K]
    w = torch.randn(N, K, device=DEV, generator=g).bfloat16()
    b = torch.randn(N, device=DEV, generator=g).bfloat16()
    want = x.double() @ w.double().T
    _close(gemm_tcgen05.gemm_nt(x, w), want, 2 ** -8)                            # one rounding to bf16: 2^-9 at most
    got = gemm_tcgen05.gemm_nt(x, w, bias=b)
    _close(got, want + b.double(), 2 ** -8)
    assert torch.equal(got, gemm_tcgen05.gemm_nt(x, w, bias=b))                 # slices meet in a fixed order


@pytest.mark.parametrize("M,I,K", [(1, 64, 128), (16, 12288, 4096), (30, 192, 2048), (64, 6144, 2048)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
def test_gated(M, I, K, act):
    g = torch.Generator(device=DEV).manual_seed(M + I)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    gate, up = ((torch.randn(I, K, device=DEV, generator=g) * K ** -0.5).bfloat16() for _ in range(2))
    got = gemm_tcgen05.gemm_act_mul(x, gemm_tcgen05.interleave_gate_up(gate, up), act)
    want = glu.apply((x.double() @ gate.double().T).bfloat16().double(), (x.double() @ up.double().T).bfloat16().double(), act)
    _close(got, want, 2 ** -7)                                                   # gate, up and their product are rounded


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(128, 128), (576, 7168), (1536, 384), (20000, 256)])
def test_fp8(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    a, a_s = fp8.quant_group128(torch.randn(M, K, device=DEV, generator=g).bfloat16())
    w, w_s = fp8.quant_block128_ref(torch.randn(N, K, device=DEV, generator=g))
    want = (a.double() * a_s.double().repeat_interleave(128, 1)) @ \
        (w.double() * w_s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).T
    _close(fp8.block_scaled_mm(a, a_s, w, w_s), want, 2 ** -8)


# more rows, in tiles of 128: rows, columns and K blocks that fill no tile, and more tiles than SMs
@pytest.mark.parametrize("M,N,K", [(130, 2048, 256), (300, 7168, 640), (922, 7168, 2048), (1000, 8200, 384), (2100, 4352, 256)])
def test_fp8_of_many_rows(M, N, K):
    test_fp8(M, N, K)


# every tile that the numbers of rows and columns choose, with K blocks that fill no stage, one slice and more of a ring, and a K
# whose scales are too many for them
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 128), (576, 7168), (1544, 384), (6400, 640), (7168, 2048), (12800, 256), (25608, 384), (128, 49280)])
def test_fp8_rows_do_not_depend_on_their_number(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    a, a_s = fp8.quant_group128(torch.randn(130, K, device=DEV, generator=g).bfloat16())
    w, w_s = fp8.quant_block128_ref(torch.randn(N, K, device=DEV, generator=g))
    assert torch.equal(fp8.block_scaled_mm(a[:M], a_s[:M], w, w_s), fp8.block_scaled_mm(a, a_s, w, w_s)[:M])


@pytest.mark.parametrize("tile", [16, 32, 64])
@pytest.mark.parametrize("N,K", [(128, 128), (384, 640), (512, 1152)])
def test_fp8_experts_rows_do_not_depend_on_the_tile(tile, N, K):
    g = torch.Generator(device=DEV).manual_seed(tile + K)
    a, a_s = fp8.quant_group128(torch.randn(256, K, device=DEV, generator=g).bfloat16())
    parts = [fp8.quant_block128_ref(torch.randn(N, K, device=DEV, generator=g)) for _ in range(2)]
    w, w_s = torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts])
    large, small = (torch.empty(256, N, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    experts = torch.tensor([1, 0], dtype=torch.int32, device=DEV)
    fp8.block_scaled_mm_grouped(a, a_s, w, w_s, experts, large, 128)
    fp8.block_scaled_mm_grouped(a, a_s, w, w_s, experts.repeat_interleave(128 // tile), small, tile)
    assert torch.equal(large, small)


@pytest.mark.parametrize("tile", [16, 32, 64, 256])
@pytest.mark.parametrize("kind", ["bf16", "gated", "fp8"])
def test_grouped(tile, kind):
    from xllm_b200.ops import _lib
    from xllm_b200.ops._lib import check, ptr, stream
    g = torch.Generator(device=DEV).manual_seed(tile)
    experts = torch.tensor([2, 0, -1, 2, 1, -1], dtype=torch.int32, device=DEV)
    if tile == 256 and kind == "fp8":
        pytest.skip("fp8 experts take tiles of up to 128 rows")
    E, N, K, M = 3, 512 if tile == 256 else 384, 640, 6 * tile
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(E, N, K, device=DEV, generator=g) * K ** -0.5).bfloat16()
    out = torch.full((M, N // 2 if kind == "gated" else N), 7.0, device=DEV, dtype=torch.bfloat16)
    if kind == "fp8":
        a, a_s = fp8.quant_group128(x)
        parts = [fp8.quant_block128_ref(w[e].float()) for e in range(E)]
        wq, w_s = torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts])
        fp8.block_scaled_mm_grouped(a, a_s, wq, w_s, experts, out, tile)
        x = a.double() * a_s.double().repeat_interleave(128, 1)
        w = torch.stack([fp8.dequant_block128_ref(q, s, torch.float64) for q, s in parts])
    elif tile == 256:
        check(_lib.load().xllm_gemm_bf16_grouped_pair(ptr(x), ptr(w), ptr(out), ptr(experts), M, N, K, E, K, out.shape[1],
                                                      int(kind == "gated"), 0.0, 0.0, stream()), "pair")
    else:
        check(_lib.load().xllm_gemm_bf16_grouped_few(ptr(x), ptr(w), ptr(out), ptr(experts), tile, M, N, K, E, K, out.shape[1],
                                                     int(kind == "gated"), 0.0, 0.0, stream()), "few")
    for i, e in enumerate(experts.tolist()):
        got = out[i * tile:(i + 1) * tile]
        if e < 0:
            assert (got == 7).all()                                              # tiles nobody has are left
            continue
        want = x[i * tile:(i + 1) * tile].double() @ w[e].double().T
        if kind == "gated":
            gate, up = want.bfloat16().double().view(tile, N // 128, 2, 64).unbind(2)
            want = glu.apply(gate, up, "silu").reshape(tile, N // 2)
        _close(got, want, 2 ** -7 if kind == "gated" else 2 ** -8)


@pytest.mark.parametrize("experts", [[1, 1, 1, 1, 0, 0, 0, 0], [0, -1, 1, 1, 0, 1, 0] + [-1] * 40, [-1] * 9])
@pytest.mark.parametrize("N,K", [(8192, 5120), (512, 4352)])
@pytest.mark.parametrize("kind", ["bf16", "pair", "fp8"])
def test_grouped_tile_orders(kind, N, K, experts):
    """Experts above what the L2 keeps, whose column tiles are swept by all row tiles, and small ones; tiles that nobody has among the
    others, behind them, and alone."""
    from xllm_b200.ops import _lib
    from xllm_b200.ops._lib import check, ptr, stream
    g = torch.Generator(device=DEV).manual_seed(N)
    E, tile = 2, 256 if kind == "pair" else 128
    experts = torch.tensor(experts, dtype=torch.int32, device=DEV)
    M = len(experts) * tile
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(E, N, K, device=DEV, generator=g) * K ** -0.5).bfloat16()
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    if kind == "fp8":
        a, a_s = fp8.quant_group128(x)
        parts = [fp8.quant_block128_ref(w[e].float()) for e in range(E)]
        fp8.block_scaled_mm_grouped(a, a_s, torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts]), experts, out)
        x = a.float() * a_s.repeat_interleave(128, 1)
        w = torch.stack([fp8.dequant_block128_ref(q, s, torch.float32) for q, s in parts])
    elif kind == "pair":
        check(_lib.load().xllm_gemm_bf16_grouped_pair(ptr(x), ptr(w), ptr(out), ptr(experts), M, N, K, E, K, N, 0, 0.0, 0.0, stream()), "pair")
    else:
        check(_lib.load().xllm_gemm_bf16_grouped(ptr(x), ptr(w), ptr(out), ptr(experts), M, N, K, E, K, N, stream()), "grouped")
    for i, e in enumerate(experts.tolist()):
        got = out[i * tile:(i + 1) * tile]
        if e < 0:
            assert (got == 7).all()
        else:
            _close(got, x[i * tile:(i + 1) * tile].double() @ w[e].double().T, 2 ** -8)


@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_grouped_with_more_tiles_than_a_grid_has_rows(kind):
    """65664 of them, as hundreds of experts with wide rows have; a grid's second and third size end at 65535."""
    from xllm_b200.ops import _lib
    from xllm_b200.ops._lib import check, ptr, stream
    g = torch.Generator(device=DEV).manual_seed(5)
    M, N, K, tile, E = 513 * 16, 128 * 128, 128, 16, 2
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(E, N, K, device=DEV, generator=g) * K ** -0.5).bfloat16()
    experts = (torch.arange(M // tile, device=DEV) % E).int()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    if kind == "fp8":
        a, a_s = fp8.quant_group128(x)
        parts = [fp8.quant_block128_ref(w[e].float()) for e in range(E)]
        fp8.block_scaled_mm_grouped(a, a_s, torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts]), experts, out, tile)
        x = a.float() * a_s.repeat_interleave(128, 1)
        w = torch.stack([fp8.dequant_block128_ref(q, s, torch.float32) for q, s in parts])
    else:
        check(_lib.load().xllm_gemm_bf16_grouped_few(ptr(x), ptr(w), ptr(out), ptr(experts), tile, M, N, K, E, K, N, 0, 0.0, 0.0,
                                                     stream()), "few")
    rows = torch.arange(M, device=DEV).view(-1, tile)
    for e in range(E):
        here = rows[experts == e].flatten()
        _close(out[here], x[here].double() @ w[e].double().T, 2 ** -8)


@pytest.mark.parametrize("rows,d,act", [(1, 128, "silu"), (48, 2048, "silu"), (33, 384, "gelu_tanh")])
def test_activation_and_its_quantisation(rows, d, act):
    from xllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(d)
    x = torch.randn(rows, 2 * d, device=DEV, generator=g).bfloat16()
    want_q, want_s = fp8.quant_group128(ops.act_and_mul(x, act))
    got_q, got_s = fp8.act_quant_group128(x, act)
    assert torch.equal(got_s, want_s) and torch.equal(got_q.view(torch.uint8), want_q.view(torch.uint8))


# (tokens, experts, chosen): one row tile after another up to pairs of CTAs, experts with more rows than a tile and with none
@pytest.mark.parametrize("T,E,K", [(1, 8, 2), (9, 32, 4), (40, 16, 4), (64, 8, 2), (130, 8, 2), (447, 8, 2), (448, 8, 2), (1500, 8, 2),
                                   (72, 16, 4), (73, 16, 4), (112, 16, 4), (113, 16, 4), (225, 16, 4), (527, 8, 2), (528, 8, 2)])
@pytest.mark.parametrize("fp8_weights", [False, True])
def test_expert_layer(T, E, K, fp8_weights):
    g = torch.Generator(device=DEV).manual_seed(T * E)
    H, I = 256, 128
    x = torch.randn(T, H, device=DEV, generator=g).bfloat16()
    logits = torch.randn(T, E, device=DEV, generator=g)
    logits[:, 1] += 3.0                                                          # a favourite
    logits[:, 2] -= 30.0                                                         # and one that nobody wants
    up, down = ((torch.randn(E, *s, device=DEV, generator=g) * s[1] ** -0.5).bfloat16() for s in ((2 * I, H), (H, I)))
    scales = None
    if fp8_weights:
        q = [[fp8.quant_block128_ref(t[e].float()) for e in range(E)] for t in (up, down)]
        scales = tuple(torch.stack([p[1] for p in parts]) for parts in q)
        qu, qd = (torch.stack([p[0] for p in parts]) for parts in q)
        up, down = (torch.stack([fp8.dequant_block128_ref(*p, torch.float32) for p in parts]) for parts in q)
    want = moe.fused_moe_reference(x, logits, up, down, K).double()
    got = moe.fused_moe(x, logits, qu if scales else up, qd if scales else down, K, w_scales=scales)
    # bf16: three roundings.  fp8: three factors of an output (gate, up through x; the activation) carry a rounding to e4m3 each,
    # uniform within 2^-4 of a value at worst, that is 2^-4 / sqrt(3) in the mean square, and independent: 2^-4 together
    _close(got, want, 2 ** -4 if scales else 2 ** -7)


_CAPTURE_FIRST = """
import torch
from xllm_b200.ops import fp8, gemm_tcgen05
x, w = (torch.randn(n, 256, device="cuda").bfloat16() for n in (96, 512))
a, a_s = fp8.quant_group128(x)
b, b_s = fp8.quant_block128_ref(w.float())
gemm_tcgen05.prepare()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    got = [gemm_tcgen05.gemm_nt(x[:4], w), fp8.block_scaled_mm(a[:4], a_s[:4], b, b_s), gemm_tcgen05.gemm_nt(x, w)]
graph.replay()
want = x.double() @ w.double().T
for y, n, rel in zip(got, (4, 4, 96), (2 ** -8, 2 ** -3, 2 ** -8)):
    assert (y.double() - want[:n]).norm() <= rel * want[:n].norm()
assert gemm_tcgen05.error_status() == 0
print("captured")
"""


def test_the_first_launches_may_be_captured():
    """prepare() leaves nothing to allocate: a process captures its first products."""
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", _CAPTURE_FIRST], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
