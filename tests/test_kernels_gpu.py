"""Each kernel alone against a plain float32 reference of the same operation, at sizes other
than the engine's: tails, odd widths, sizes that are no power of two."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def status():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def rand(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


# ------------------------------------------------------------------------------- elementwise
@pytest.mark.parametrize("table_dtype", [torch.float32, torch.bfloat16])
def test_embed(status, table_dtype):
    from sprout_lm_b200 import kernels
    table = rand(101, 72, dtype=table_dtype)
    tokens = torch.tensor([0, 100, 5, 5, 37], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 72, dtype=torch.float32, device=DEV)
    kernels.embed(table, tokens, out, status)
    assert torch.equal(out, table[tokens.long()].float())
    assert int(status.item()) == 0
    bad = torch.tensor([3, 101], dtype=torch.int32, device=DEV)
    kernels.embed(table, bad, out[:2], status)                    # flagged, not faulted
    assert int(status.item()) & 2
    status.zero_()


@pytest.mark.parametrize("hidden,eps", [(72, 1e-6), (896, 1e-5), (1000, 1e-6), (4100, 1e-5)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm(hidden, eps, out_dtype):
    from sprout_lm_b200 import kernels
    x = rand(7, hidden, scale=3.0)
    gain = 1 + rand(hidden, scale=0.1, seed=1)
    out = torch.empty(7, hidden, dtype=out_dtype, device=DEV)
    kernels.rmsnorm(x, gain, out, eps)
    x64 = x.double()
    want = (x64 / torch.sqrt((x64 * x64).mean(-1, keepdim=True) + eps)).float().double() * gain.double()
    tol = 2e-6 if out_dtype == torch.float32 else 8e-3
    assert (out.double() - want).abs().max().item() <= tol * want.abs().max().item()
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    picked = torch.empty(3, hidden, dtype=out_dtype, device=DEV)
    kernels.rmsnorm(x, gain, picked, eps, rows)
    assert torch.equal(picked, out[rows.long()])


@pytest.mark.parametrize("hidden", [72, 896, 1000, 2048])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm_many_rows(hidden, out_dtype):
    """A prefill's worth of rows takes the warp-per-row kernel: the same numbers as the
    block-per-row kernel gives for a few rows, to the last bit of the output's rounding."""
    from sprout_lm_b200 import kernels
    rows, eps = 203, 1e-6
    x = rand(rows, hidden, scale=3.0, seed=4)
    gain = 1 + rand(hidden, scale=0.1, seed=1)
    out = torch.empty(rows, hidden, dtype=out_dtype, device=DEV)
    kernels.rmsnorm(x, gain, out, eps)
    x64 = x.double()
    want = (x64 / torch.sqrt((x64 * x64).mean(-1, keepdim=True) + eps)).float().double() * gain.double()
    tol = 2e-6 if out_dtype == torch.float32 else 8e-3
    assert (out.double() - want).abs().max().item() <= tol * want.abs().max().item()
    few = torch.empty(5, hidden, dtype=out_dtype, device=DEV)
    kernels.rmsnorm(x[100:105].contiguous(), gain, few, eps)
    assert (few.double() - out[100:105].double()).abs().max().item() <= tol * want.abs().max().item()


@pytest.mark.parametrize("heads,kv_heads,head_dim,page,theta", [(14, 2, 64, 16, 1e6), (8, 2, 128, 32, 1e4), (4, 2, 16, 8, 1e4), (3, 1, 48, 16, 1e5)])
@pytest.mark.parametrize("rotate", [True, False])
def test_rope_append_many_tokens(status, heads, kv_heads, head_dim, page, theta, rotate):
    """A prefill's worth of tokens takes the vectorised kernel (bfloat16): checked against the
    float64 rotation and against the cache slots that the block tables name."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    dtype = torch.bfloat16
    lengths = [97, 3, 130]                                   # tokens of three requests, from position 5, 0 and 40
    starts = [5, 0, 40]
    pages_each = [-(-(s0 + n) // page) for s0, n in zip(starts, lengths)]
    pool = sum(pages_each) + 2
    perm = torch.randperm(pool, generator=torch.Generator().manual_seed(3)).to(torch.int32)
    table = torch.full((3, max(pages_each)), -1, dtype=torch.int32)
    at = 0
    for r, n in enumerate(pages_each):
        table[r, :n] = perm[at:at + n]
        at += n
    positions = torch.cat([torch.arange(s0, s0 + n, dtype=torch.int32) for s0, n in zip(starts, lengths)])
    seq_of_token = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(lengths)])
    T = positions.numel()

    class RT:
        device = torch.device(DEV)
    cos, sin = HalfSplitRotary("", head_dim, theta, 512).rotary_tables(RT) if rotate else (None, None)
    width = (heads + 2 * kv_heads) * head_dim
    qkv = rand(T, width, dtype=dtype, seed=8)
    original = qkv.clone()
    k_cache = torch.zeros(pool, kv_heads, page, head_dim, dtype=dtype, device=DEV)
    v_cache = torch.zeros_like(k_cache)
    kernels.rope_append(qkv, positions.to(DEV), seq_of_token.to(DEV), table.to(DEV), cos, sin, k_cache, v_cache,
                        heads, kv_heads, head_dim, page, True, status)
    assert int(status.item()) == 0
    q0, k0 = original[:, :heads * head_dim], original[:, heads * head_dim:(heads + kv_heads) * head_dim]
    q_want = rope_reference(q0, positions, head_dim, theta) if rotate else q0.double().cpu()
    k_want = rope_reference(k0, positions, head_dim, theta) if rotate else k0.double().cpu()
    assert (qkv[:, :heads * head_dim].double().cpu() - q_want).abs().max().item() <= 6.4e-2
    assert torch.equal(qkv[:, heads * head_dim:], original[:, heads * head_dim:])       # k and v stay in qkv as projected
    pg = table[seq_of_token.long(), (positions // page).long()].long()
    slot = (positions % page).long()
    got_k = k_cache[pg.to(DEV), :, slot.to(DEV), :].reshape(T, -1).double().cpu()
    assert (got_k - k_want).abs().max().item() <= 6.4e-2
    assert torch.equal(v_cache[pg.to(DEV), :, slot.to(DEV), :].reshape(T, -1), original[:, (heads + kv_heads) * head_dim:])
    assert int((k_cache != 0).any(-1).any(1).sum().item()) == T                      # no other slot was touched
    # the few-token kernel gives the same bits
    few_q = original[:6].clone()
    k2, v2 = torch.zeros_like(k_cache), torch.zeros_like(v_cache)
    kernels.rope_append(few_q, positions[:6].to(DEV), seq_of_token[:6].to(DEV), table.to(DEV), cos, sin, k2, v2,
                        heads, kv_heads, head_dim, page, True, status)
    assert torch.equal(few_q, qkv[:6])
    assert torch.equal(k2[pg[:6].to(DEV), :, slot[:6].to(DEV), :], k_cache[pg[:6].to(DEV), :, slot[:6].to(DEV), :])
    # the same from float32 sums plus a bias (what a split-K product leaves): the rotated q lands in
    # qkv, k and v in the cache, the sums are cleared
    bias = rand(width, seed=9)
    acc = torch.zeros(T + 2, width, device=DEV)
    acc[:T] = original.float() - bias
    out_q = torch.zeros_like(original)
    k4, v4 = torch.zeros_like(k_cache), torch.zeros_like(v_cache)
    kernels.rope_append(out_q, positions.to(DEV), seq_of_token.to(DEV), table.to(DEV), cos, sin, k4, v4,
                        heads, kv_heads, head_dim, page, True, status, acc=acc[:T], bias=bias)
    assert (out_q[:, :heads * head_dim].float() - qkv[:, :heads * head_dim].float()).abs().max().item() <= 2e-2
    assert (k4.float() - k_cache.float()).abs().max().item() <= 2e-2
    assert (v4.float() - v_cache.float()).abs().max().item() <= 2e-2
    assert float(acc.abs().max()) == 0.0
    assert int((k4 != 0).any(-1).any(1).sum().item()) == T
    # without the cache write only q changes
    k3 = torch.zeros_like(k_cache)
    only_q = original.clone()
    kernels.rope_append(only_q, positions.to(DEV), seq_of_token.to(DEV), table.to(DEV), cos, sin, k3, v2.zero_(),
                        heads, kv_heads, head_dim, page, False, status)
    assert torch.equal(only_q, qkv) and float(k3.abs().max()) == 0.0 and float(v2.abs().max()) == 0.0
    assert int(status.item()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inter", [8, 320, 4864])
def test_swiglu_interleaved(dtype, inter):
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.mlp import interleave_gate_up
    gate, up = rand(5, inter, dtype=dtype, scale=2.0), rand(5, inter, dtype=dtype, scale=2.0, seed=3)
    fused = interleave_gate_up(gate.T.contiguous(), up.T.contiguous()).T.contiguous()   # columns interleaved like weight rows
    out = torch.empty(5, inter, dtype=dtype, device=DEV)
    kernels.swiglu(fused, out)
    g = gate.double()
    want = (g / (1 + torch.exp(-g))).float().double() * up.double()
    tol = 1e-6 if dtype == torch.float32 else 8e-3
    assert (out.double() - want).abs().max().item() <= tol * max(1.0, want.abs().max().item())
    with pytest.raises(kernels.KernelError, match="multiple of 8"):
        kernels.swiglu(torch.empty(2, 24, dtype=dtype, device=DEV), torch.empty(2, 12, dtype=dtype, device=DEV))


def rope_reference(x, positions, head_dim, theta):
    tokens = x.shape[0]
    heads = x.shape[1] // head_dim
    half = head_dim // 2
    d = torch.arange(half, dtype=torch.float64)
    angle = positions.double()[:, None, None] / theta ** (2 * d / head_dim)[None, None, :]
    xs = x.double().cpu().reshape(tokens, heads, head_dim)
    a, b = xs[..., :half], xs[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1).reshape(tokens, -1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,theta", [(4, 2, 16, 16, 1e4), (3, 1, 32, 8, 1e6), (5, 5, 48, 4, 5e5), (14, 2, 64, 16, 1e6)])
def test_rope_append(status, dtype, heads, kv_heads, head_dim, page, theta):
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    max_pos, pages = 4096, 40
    rotary = HalfSplitRotary("", head_dim, theta, max_pos)

    class RT:
        device = torch.device(DEV)
    cos, sin = rotary.rotary_tables(RT)
    positions = torch.tensor([0, 1, page - 1, page, 3 * page + 1, 4095 % (pages * page // 2)], dtype=torch.int32)
    T = positions.numel()
    # two requests with scattered pages
    seq_of_token = torch.tensor([0, 0, 0, 1, 1, 1], dtype=torch.int32)
    max_pages = pages // 2
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).to(torch.int32)
    table = perm.reshape(2, max_pages).contiguous()
    width = (heads + 2 * kv_heads) * head_dim
    qkv = rand(T, width, dtype=dtype)
    original = qkv.clone()
    k_cache = torch.zeros(pages, kv_heads, page, head_dim, dtype=dtype, device=DEV)
    v_cache = torch.zeros_like(k_cache)
    kernels.rope_append(qkv, positions.to(DEV), seq_of_token.to(DEV), table.to(DEV), cos, sin, k_cache, v_cache,
                        heads, kv_heads, head_dim, page, True, status)
    assert int(status.item()) == 0
    q_want = rope_reference(original[:, :heads * head_dim], positions, head_dim, theta)
    k_want = rope_reference(original[:, heads * head_dim:(heads + kv_heads) * head_dim], positions, head_dim, theta)
    tol = 2e-6 if dtype == torch.float32 else 1.6e-2
    assert (qkv[:, :heads * head_dim].double().cpu() - q_want).abs().max().item() <= tol * 4
    for t in range(T):
        pos = int(positions[t])
        pg, slot = int(table[seq_of_token[t], pos // page]), pos % page
        got_k = k_cache[pg, :, slot, :].reshape(-1).double().cpu()
        assert (got_k - k_want[t]).abs().max().item() <= tol * 4
        got_v = v_cache[pg, :, slot, :].reshape(-1)
        assert torch.equal(got_v, original[t, (heads + kv_heads) * head_dim:])
    # nothing else was touched
    assert int((k_cache != 0).any(-1).any(1).sum().item()) == T
    # the same from float32 sums plus a bias (what a split-K product leaves): same rotation, the
    # rotated q lands in qkv, the sums are cleared
    bias = rand(width, seed=9)
    acc = torch.zeros(T + 2, width, device=DEV)
    acc[:T] = original.float() - bias
    out_q = torch.zeros_like(original)
    k2, v2 = torch.zeros_like(k_cache), torch.zeros_like(v_cache)
    kernels.rope_append(out_q, positions.to(DEV), seq_of_token.to(DEV), table.to(DEV), cos, sin, k2, v2,
                        heads, kv_heads, head_dim, page, True, status, acc=acc[:T], bias=bias)
    slack = 1e-5 if dtype == torch.float32 else 2e-2
    assert (out_q[:, :heads * head_dim].float() - qkv[:, :heads * head_dim].float()).abs().max().item() <= slack
    assert (k2.float() - k_cache.float()).abs().max().item() <= slack
    assert (v2.float() - v_cache.float()).abs().max().item() <= slack
    assert float(acc.abs().max()) == 0.0
    # a page id outside the pool is flagged and skipped
    bad = table.clone()
    bad[0, 0] = pages + 3
    kernels.rope_append(original.clone(), positions.to(DEV), seq_of_token.to(DEV), bad.to(DEV), cos, sin, k_cache,
                        v_cache, heads, kv_heads, head_dim, page, True, status)
    assert int(status.item()) & 1
    status.zero_()


# ------------------------------------------------------------------------------- matrix products
SHAPES = [(1, 1, 8), (1, 896, 896), (3, 130, 72), (8, 1152, 896), (17, 509, 96), (64, 256, 4864), (100, 77, 200),
          (128, 896, 896), (129, 300, 136), (257, 1000, 328), (600, 1152, 896), (2048, 896, 4864), (300, 512, 200),
          (1100, 1024, 896)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_simple_float32(M, N, K):
    from sprout_lm_b200 import kernels
    a, w, bias = rand(M, K), rand(N, K, seed=1), rand(N, seed=2)
    out = torch.empty(M, N, device=DEV)
    kernels.gemm_simple(a, w, out, bias=bias)
    want = a.double() @ w.double().T + bias.double()
    # sequential float32 accumulation: error grows like eps * sqrt(K) times the magnitude of the sums
    tol = 4 * 6e-8 * math.sqrt(K) * want.abs().max().item() + 1e-6
    assert (out.double() - want).abs().max().item() <= tol
    # a row's result does not depend on the rows around it
    if M > 2:
        alone = torch.empty(1, N, device=DEV)
        kernels.gemm_simple(a[M // 2:M // 2 + 1], w, alone, bias=bias)
        assert torch.equal(alone[0], out[M // 2])
    x = rand(M, N, seed=5)
    want = x.double() + a.double() @ w.double().T
    kernels.gemm_simple(a, w, x, residual=x)
    assert (x.double() - want).abs().max().item() <= tol


@pytest.mark.parametrize("M,N,K", [(8, 129, 33), (9, 257, 36), (16, 130, 63), (17, 65, 31), (65, 63, 100), (1153, 8390, 37), (1153, 8390, 40)])
def test_gemm_simple_tiles(M, N, K):
    """Sizes at the edges of every tile and of the 16-byte loads: a row's bits do not depend on the tile its call's sizes pick."""
    from sprout_lm_b200 import kernels
    a, w = rand(M, K), rand(N, K, seed=1)
    out = torch.empty(M, N, device=DEV)
    kernels.gemm_simple(a, w, out)
    want = a.double() @ w.double().T
    tol = 4 * 6e-8 * math.sqrt(K) * want.abs().max().item() + 1e-6      # sequential float32 accumulation
    assert (out.double() - want).abs().max().item() <= tol
    for first, rows in ((M - 1, 1), (0, min(M, 16)), (0, min(M, 17))):
        part = torch.empty(rows, N, device=DEV)
        kernels.gemm_simple(a[first:first + rows], w, part)
        assert torch.equal(part, out[first:first + rows])


@pytest.mark.parametrize("M,N,K", [(8, 129, 256), (16, 65, 300), (17, 200, 4099), (130, 4097, 257), (64, 4096, 1000), (1153, 63, 260), (700, 2048, 256)])
def test_gemm_simple_shares_of_k(M, N, K):
    """K shared by a cluster's CTAs (in four or eight up to 4,096 columns, in two beyond), at ragged ends of rows, columns and shares, on and off 16-byte rows:
    a row's bits depend neither on the rows beside it nor on the tile; strided output, bias and residual."""
    from sprout_lm_b200 import kernels
    a, w, bias = rand(M, K), rand(N, K, seed=1), rand(N, seed=2)
    out = torch.empty(M, N, device=DEV)
    kernels.gemm_simple(a, w, out, bias=bias)
    want = a.double() @ w.double().T + bias.double()
    tol = 4 * 6e-8 * math.sqrt(K) * want.abs().max().item() + 1e-6      # sequential float32 accumulation; shares only shorten it
    assert (out.double() - want).abs().max().item() <= tol
    for first, rows in ((M - 1, 1), (0, min(M, 16)), (0, min(M, 17)), (0, min(M, 65))):
        part = torch.empty(rows, N, device=DEV)
        kernels.gemm_simple(a[first:first + rows], w, part, bias=bias)
        assert torch.equal(part, out[first:first + rows])
    for lead in (1, 4):
        wide = torch.full((M, N + 2 * lead), 2.0, device=DEV)
        x = wide[:, lead:lead + N]
        kernels.gemm_simple(a, w, x, bias=bias, residual=x)
        assert torch.equal(x, out + 2.0) and (wide[:, :lead] == 2.0).all() and (wide[:, lead + N:] == 2.0).all()


@pytest.mark.parametrize("M,N,K", [(1, 70, 4097), (17, 900, 4100), (64, 1030, 4864), (130, 66, 8190)])
def test_gemm_simple_eight_shares_of_k(M, N, K):
    """K shared by the eight CTAs of a cluster (from 4,096 on, up to 4,096 columns), the last shares short or empty."""
    test_gemm_simple_shares_of_k(M, N, K)


@pytest.mark.parametrize("orientation", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_bf16_tensor_cores(status, M, N, K, orientation):
    """orientation 0: the kernel's own choice; 1: tokens on the MMA's M axis; 2: weight rows on M;
    3: tokens on M with single CTAs; 4: with CTA pairs (tcgen05.mma.cta_group::2)."""
    from sprout_lm_b200 import kernels
    a, w, bias = rand(M, K, dtype=torch.bfloat16), rand(N, K, dtype=torch.bfloat16, seed=1), rand(N, seed=2)
    want = a.double() @ w.double().T + bias.double()
    scale = want.abs().max().item()
    out = torch.full((M, N), float("nan"), dtype=torch.float32, device=DEV)
    kernels.gemm_bf16(a, w, out, status, bias=bias, orientation=orientation)
    assert (out.double() - want).abs().max().item() <= 1e-5 * scale + 1e-6       # float32 accumulation of exact products
    out16 = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_bf16(a, w, out16, status, bias=bias, orientation=orientation)
    assert (out16.double() - want).abs().max().item() <= 8e-3 * scale
    x = rand(M, N, seed=5)
    want_res = x.double() + a.double() @ w.double().T
    kernels.gemm_bf16(a, w, x, status, residual=x, orientation=orientation)
    assert (x.double() - want_res).abs().max().item() <= 1e-5 * scale + 1e-6
    assert int(status.item()) == 0


@pytest.mark.parametrize("orientation", [0, 2, 3, 4])
@pytest.mark.parametrize("M,inter,K", [(5, 200, 72), (300, 256, 136), (2048, 384, 896), (513, 4864, 96),
                                       (64, 640, 200), (65, 640, 200), (100, 4864, 896), (128, 256, 136), (129, 768, 72), (200, 4864, 96)])
def test_gemm_bf16_swiglu_epilogue(status, M, inter, K, orientation):
    """gate and up rows interleaved in blocks of 8; the epilogue writes silu(gate) * up.  The sizes
    lie on both sides of the token counts at which the arrangement changes (64, 128, 256)."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.mlp import interleave_gate_up
    if orientation == 2 and M > 256:
        pytest.skip("weights on M takes up to 256 tokens")
    a = rand(M, K, dtype=torch.bfloat16)
    gate, up = rand(inter, K, dtype=torch.bfloat16, seed=1), rand(inter, K, dtype=torch.bfloat16, seed=2)
    w = interleave_gate_up(gate, up)
    out = torch.full((M, inter), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_bf16(a, w, out, status, swiglu=True, orientation=orientation)
    g, u = a.double() @ gate.double().T, a.double() @ up.double().T
    want = g / (1 + torch.exp(-g)) * u
    assert (out.double() - want).abs().max().item() <= 8e-3 * max(1.0, want.abs().max().item())
    assert int(status.item()) == 0


@pytest.mark.parametrize("kind", ["bfloat16", "float32", "residual", "swiglu"])
@pytest.mark.parametrize("orientation", [3, 4])
@pytest.mark.parametrize("M,N,K,lead,extra", [(257, 272, 72, 0, 0), (300, 528, 136, 8, 8), (129, 1344, 200, 1, 3), (513, 224, 264, 0, 5), (260, 96, 64, 2, 2)])
def test_gemm_bf16_tokens_on_m_stores_rows(status, kind, orientation, M, N, K, lead, extra):
    """The epilogues with tokens on M go through a warp's shared memory in rows of 128 bytes: outputs that are columns of a wider buffer, on and off
    16-byte boundaries, ragged last tiles of rows and columns; what lies beside the output stays as it was."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.mlp import interleave_gate_up
    a, bias = rand(M, K, dtype=torch.bfloat16), rand(N, seed=2)
    cols, dtype = (N // 2, torch.bfloat16) if kind == "swiglu" else (N, torch.bfloat16 if kind == "bfloat16" else torch.float32)
    if kind == "swiglu" and (lead + cols + extra) % 2:
        extra += 1                                             # that epilogue takes even row strides
    buffer = torch.full((M, lead + cols + extra), 3.0, dtype=dtype, device=DEV)
    out = buffer[:, lead:lead + cols]
    if kind == "swiglu":
        gate, up = rand(cols, K, dtype=torch.bfloat16, seed=1), rand(cols, K, dtype=torch.bfloat16, seed=4)
        kernels.gemm_bf16(a, interleave_gate_up(gate, up), out, status, swiglu=True, orientation=orientation)
        g = a.double() @ gate.double().T
        want = g / (1 + torch.exp(-g)) * (a.double() @ up.double().T)
    else:
        w = rand(N, K, dtype=torch.bfloat16, seed=1)
        kernels.gemm_bf16(a, w, out, status, bias=bias, residual=out if kind == "residual" else None, orientation=orientation)
        want = a.double() @ w.double().T + bias.double() + (3.0 if kind == "residual" else 0.0)
    # float32 sums of exact products; a bfloat16 output is rounded by up to 2^-9 of its value (twice that, and the activation, with a gate)
    tol = 1e-5 if dtype == torch.float32 else 8e-3
    assert (out.double() - want).abs().max().item() <= tol * max(1.0, want.abs().max().item())
    assert (buffer[:, :lead] == 3.0).all() and (buffer[:, lead + cols:] == 3.0).all()
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,N,K,residual", [(2048, 1152, 896, False), (2048, 1344, 2048, False), (2048, 896, 4864, True), (2048, 2048, 2048, True),
                                            (2048, 3072, 2048, False), (2500, 8224, 1024, False), (4001, 3088, 1024, False), (600, 896, 4864, True),
                                            (2049, 900, 4864, True)])
def test_gemm_bf16_token_tiles_of_every_form(status, M, N, K, residual):
    """Sizes whose tiles the kernel picks among all forms: single CTAs of 128, 192, 224 and 256 columns, pairs of 192, 224 and 256, K divided where the
    output is added to, last tiles that reach beyond the matrix."""
    from sprout_lm_b200 import kernels
    a, w = rand(M, K, dtype=torch.bfloat16), rand(N, K, dtype=torch.bfloat16, seed=1)
    buffer = torch.full((M, N + 4), 2.0 if residual else float("nan"), device=DEV)
    out = buffer[:, :N]
    kernels.gemm_bf16(a, w, out, status, residual=out if residual else None)
    want = a.double() @ w.double().T + (2.0 if residual else 0.0)
    assert (out.double() - want).abs().max().item() <= 1e-5 * want.abs().max().item()       # float32 sums of exact products
    assert torch.equal(buffer[:, N:], torch.full((M, 4), 2.0, device=DEV)) if residual else bool(buffer[:, N:].isnan().all())
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,N,K,split", [(1, 896, 4864, 16), (8, 896, 896, 14), (64, 130, 1000, 5), (128, 256, 264, 9)])
def test_gemm_bf16_split_k(status, M, N, K, split):
    from sprout_lm_b200 import kernels
    a, w = rand(M, K, dtype=torch.bfloat16), rand(N, K, dtype=torch.bfloat16, seed=1)
    x = rand(M, N, seed=5)
    want = x.double() + a.double() @ w.double().T
    kernels.gemm_bf16(a, w, x, status, residual=x, orientation=2, split_k=split)
    assert (x.double() - want).abs().max().item() <= 2e-5 * want.abs().max().item() + 1e-6
    assert int(status.item()) == 0


@pytest.mark.parametrize("tokens,hidden,inter,eps", [(1, 64, 128, 1e-6), (5, 96, 320, 1e-5), (8, 896, 4864, 1e-6),
                                                     (3, 1024, 2816, 1e-5), (8, 1536, 2048, 1e-6), (2, 48, 16, 1e-6),
                                                     (9, 896, 4864, 1e-6), (16, 896, 4864, 1e-6), (13, 96, 320, 1e-5),
                                                     (11, 1024, 2816, 1e-5), (16, 48, 16, 1e-6)])
def test_ffn_decode_one_kernel(status, tokens, hidden, inter, eps):
    """RMSNorm, gate/up, SwiGLU, down and the residual sum in one launch, against the same
    arithmetic in float64 with the kernel's two roundings to bfloat16 (the normalised rows, the
    activation).  Three launches in a row, and one channel of the input is made large so that a
    wrong row or column of any operand shows."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.mlp import interleave_gate_up
    assert kernels.ffn_decode_supported(tokens, hidden, inter)
    gate, up = rand(inter, hidden, dtype=torch.bfloat16, scale=0.05, seed=1), rand(inter, hidden, dtype=torch.bfloat16, scale=0.05, seed=2)
    down = rand(hidden, inter, dtype=torch.bfloat16, scale=0.05, seed=3)
    gain = 1 + rand(hidden, scale=0.1, seed=4)
    w = interleave_gate_up(gate, up)
    for round_ in range(3):
        x = rand(tokens, hidden, seed=10 + round_)
        x[:, (7 * round_ + 3) % hidden] *= 6.0
        h = x.double() / torch.sqrt((x.double() ** 2).mean(dim=1, keepdim=True) + eps) * gain.double()
        h = h.float().to(torch.bfloat16).double()
        g, u = h @ gate.double().T, h @ up.double().T
        t = (g / (1 + torch.exp(-g)) * u).float().to(torch.bfloat16).double()
        delta = t @ down.double().T
        want = x.double() + delta
        kernels.ffn_decode(x, gain, eps, w, down, status)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        assert (x.double() - want).abs().max().item() <= 4e-3 * max(1e-3, delta.abs().max().item())


def test_ffn_decode_refuses_what_does_not_fit(status):
    from sprout_lm_b200 import kernels
    assert not kernels.ffn_decode_supported(17, 896, 4864)         # more tokens than two tiles have columns
    assert not kernels.ffn_decode_supported(8, 904, 4864)          # sizes that are no multiple of 16
    assert not kernels.ffn_decode_supported(8, 3584, 18944)        # a CTA's share exceeds shared memory
    x = rand(8, 3584)
    with pytest.raises(kernels.KernelError, match="ffn_decode"):
        kernels.ffn_decode(x, rand(3584), 1e-6, rand(2 * 18944, 3584, dtype=torch.bfloat16), rand(3584, 18944, dtype=torch.bfloat16), status)


@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("tokens,N,K", [(1, 128, 64), (8, 1152, 896), (5, 160, 96), (8, 896, 896), (3, 48, 16), (7, 2048, 1536),
                                        (9, 1152, 896), (16, 896, 896), (12, 160, 96), (16, 48, 16), (10, 2048, 1536)])
def test_linear_decode_small_batch(status, tokens, N, K, normed):
    """out += input W^T for a few tokens with light CTAs; the input is bfloat16 rows or the RMSNorm
    of float32 rows computed inside the kernel.  The sums land on what the output held before."""
    from sprout_lm_b200 import kernels
    assert kernels.linear_decode_supported(tokens, N, K)
    w = rand(N, K, dtype=torch.bfloat16, scale=0.05, seed=1)
    before = rand(tokens, N, seed=2)
    for round_ in range(2):
        out = before.clone()
        if normed:
            x, gain, eps = rand(tokens, K, seed=3 + round_), 1 + rand(K, scale=0.1, seed=4), 1e-5
            x[:, (5 * round_ + 2) % K] *= 6.0
            h = x.double() / torch.sqrt((x.double() ** 2).mean(dim=1, keepdim=True) + eps) * gain.double()
            h = h.float().to(torch.bfloat16).double()
            kernels.linear_decode(w, out, status, norm=(x, gain, eps))
        else:
            a = rand(tokens, K, dtype=torch.bfloat16, seed=3 + round_)
            h = a.double()
            kernels.linear_decode(w, out, status, a=a)
        delta = h @ w.double().T
        # a normalised value may round to the neighbouring bfloat16 where the row's sum differs in order
        bound = (4e-3 if normed else 2e-5) * max(1e-3, delta.abs().max().item()) + 1e-6
        assert (out.double() - (before.double() + delta)).abs().max().item() <= bound
    assert int(status.item()) == 0


def test_linear_decode_refuses_what_does_not_fit(status):
    from sprout_lm_b200 import kernels
    assert not kernels.linear_decode_supported(17, 896, 896)
    assert not kernels.linear_decode_supported(8, 900, 896)
    assert not kernels.linear_decode_supported(8, 3584, 3584)       # pieces too large for light CTAs
    with pytest.raises(kernels.KernelError, match="linear_decode"):
        kernels.linear_decode(rand(3584, 3584, dtype=torch.bfloat16), rand(8, 3584), status, a=rand(8, 3584, dtype=torch.bfloat16))


@pytest.mark.parametrize("tokens,N,K,split", [(17, 1152, 896, 14), (64, 1152, 896, 14), (33, 256, 136, 3), (200, 384, 520, 9), (64, 1152, 896, 1),
                                              (64, 4608, 3584, 4), (40, 256, 2000, 1), (130, 300, 3000, 2), (8, 20000, 64, 1)])
def test_gemm_bf16_unscaled_is_the_normed_product_without_its_scale(status, tokens, N, K, split):
    """out += bfloat16(x * gain) W^T with the tokens' tiles made inside the kernel: against float64
    with that one rounding, on top of what the output held; and scaled by 1 / rms(x) it is the
    product of the RMSNorm's output, to bfloat16's precision.  K ranges of 14, 32 and 24 k-blocks per
    CTA go round the ring of stages more than once."""
    from sprout_lm_b200 import kernels
    if not kernels.gemm_bf16_unscaled_supported(tokens, N, K, split):
        assert N == 20000                                  # more work items than SMs (K ranges longer than the ring are taken)
        with pytest.raises(kernels.KernelError, match="gemm_bf16_unscaled"):
            kernels.gemm_bf16_unscaled(rand(tokens, K), rand(K), rand(N, K, dtype=torch.bfloat16), rand(tokens, N), status, split_k=split)
        return
    x = rand(tokens, K, seed=1)
    x[:, 5 % K] *= 6.0
    gain = 1 + rand(K, scale=0.1, seed=2)
    w = rand(N, K, dtype=torch.bfloat16, scale=0.05, seed=3)
    before = rand(tokens, N, seed=4)
    out = before.clone()
    for _ in range(2):                                     # twice: the sums add up
        kernels.gemm_bf16_unscaled(x, gain, w, out, status, split_k=split)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    h = (x.double() * gain.double()).float().to(torch.bfloat16).double()
    want = before.double() + 2 * (h @ w.double().T)
    assert (out.double() - want).abs().max().item() <= 2e-5 * max(1.0, want.abs().max().item())
    eps = 1e-5
    inv = 1.0 / torch.sqrt((x.double() ** 2).mean(dim=1, keepdim=True) + eps)
    normed = (x.double() * inv * gain.double()).float().to(torch.bfloat16).double() @ w.double().T
    scaled = (out.double() - before.double()) / 2 * inv
    assert (scaled - normed).abs().max().item() <= 8e-3 * max(1e-3, normed.abs().max().item())


def test_gemm_bf16_refuses_unaligned_rows(status):
    from sprout_lm_b200 import kernels
    a, w = rand(4, 20, dtype=torch.bfloat16), rand(8, 20, dtype=torch.bfloat16)
    with pytest.raises(kernels.KernelError, match="multiples of 8"):
        kernels.gemm_bf16(a, w, torch.empty(4, 8, device=DEV), status)


# ------------------------------------------------------------------------------- attention
def attention_reference(q, keys, values, heads, kv_heads, head_dim):
    """q [heads*hd]; keys, values [n, kv_heads*hd] (float64) -> [heads*hd]."""
    out = torch.zeros(heads * head_dim, dtype=torch.float64)
    group = heads // kv_heads
    for h in range(heads):
        g = h // group
        s = keys[:, g * head_dim:(g + 1) * head_dim] @ q[h * head_dim:(h + 1) * head_dim] / math.sqrt(head_dim)
        out[h * head_dim:(h + 1) * head_dim] = torch.softmax(s, 0) @ values[:, g * head_dim:(g + 1) * head_dim]
    return out


def build_paged_case(dtype, heads, kv_heads, head_dim, page, lengths, q_counts, seed=0, spike=None, poison=False,
                     layout="scattered"):
    """Requests with ``lengths`` cached positions each (the last ``q_counts`` of them are this
    step's queries), in pages scattered over the pool (``layout`` "runs": in runs of 1 to 11 pages
    that follow one another in the pool, the runs scattered; "in order": as a fresh pool hands
    them out).  ``poison``: every slot that holds no key of a request (the rest of a last page,
    pages nobody owns) is NaN instead of zero."""
    g = torch.Generator().manual_seed(seed)
    R = len(lengths)
    pages_each = [-(-n // page) for n in lengths]
    pool = sum(pages_each) + 3
    if layout == "scattered":
        order = torch.randperm(pool, generator=g)
    elif layout == "in order":
        order = torch.arange(pool)
    else:
        runs, at = [], 0
        while at < pool:
            n = min(pool - at, int(torch.randint(1, 12, (1,), generator=g)))
            runs.append(torch.arange(at, at + n))
            at += n
        order = torch.cat([runs[i] for i in torch.randperm(len(runs), generator=g)])
    table = torch.full((R, max(pages_each)), -1, dtype=torch.int32)
    k_cache = torch.full((pool, kv_heads, page, head_dim), float("nan") if poison else 0.0)
    v_cache = torch.full((pool, kv_heads, page, head_dim), float("nan") if poison else 0.0)
    keys, values, at = [], [], 0
    for r, n in enumerate(lengths):
        k = torch.randn(n, kv_heads * head_dim, generator=g)
        v = torch.randn(n, kv_heads * head_dim, generator=g)
        if spike is not None and r == spike[0]:
            k[spike[1]] *= 6.0                       # one far key whose score stands out
        k, v = k.to(dtype).float(), v.to(dtype).float()
        keys.append(k.double())
        values.append(v.double())
        for i in range(pages_each[r]):
            pg = int(order[at]); at += 1
            table[r, i] = pg
            rows = slice(i * page, min(n, (i + 1) * page))
            count = rows.stop - rows.start
            k_cache[pg, :, :count] = k[rows].reshape(count, kv_heads, head_dim).transpose(0, 1)
            v_cache[pg, :, :count] = v[rows].reshape(count, kv_heads, head_dim).transpose(0, 1)
    positions, seq_of_token = [], []
    for r, (n, c) in enumerate(zip(lengths, q_counts)):
        positions += list(range(n - c, n))
        seq_of_token += [r] * c
    T = len(positions)
    q = torch.randn(T, heads * head_dim, generator=g)
    if spike is not None:
        # queries of the spiked request look at the spiked key
        for t in range(T):
            if seq_of_token[t] == spike[0]:
                group = heads // kv_heads
                for h in range(heads):
                    gk = h // group
                    q[t, h * head_dim:(h + 1) * head_dim] = keys[spike[0]][spike[1], gk * head_dim:(gk + 1) * head_dim].float()
    q = q.to(dtype)
    want = torch.stack([attention_reference(q[t].double(), keys[seq_of_token[t]][:positions[t] + 1],
                                            values[seq_of_token[t]][:positions[t] + 1], heads, kv_heads, head_dim)
                        for t in range(T)])
    dev = lambda x, dt=None: x.to(dt or x.dtype).to(DEV)
    return dict(q=dev(q), k_cache=dev(k_cache, dtype), v_cache=dev(v_cache, dtype), table=dev(table),
                positions=dev(torch.tensor(positions, dtype=torch.int32)),
                seq_of_token=dev(torch.tensor(seq_of_token, dtype=torch.int32)), want=want, T=T,
                q_start=dev(torch.tensor(np.cumsum([0] + list(q_counts)), dtype=torch.int32)),
                context_lens=dev(torch.tensor(lengths, dtype=torch.int32)), lengths=lengths, q_counts=q_counts)


ATTN_CASES = [
    # heads, kv_heads, head_dim, page, cached lengths, queries of this step
    (4, 2, 16, 16, [5, 17, 33], [5, 1, 33]),
    (3, 1, 32, 8, [61, 1, 130], [7, 1, 1]),
    (14, 2, 64, 16, [300, 129, 16], [1, 1, 16]),
    (5, 5, 48, 4, [40, 9], [2, 9]),
    (8, 2, 128, 16, [257, 64], [3, 64]),
    (6, 3, 80, 32, [100], [100]),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths,q_counts", ATTN_CASES)
def test_attention_simple(status, dtype, heads, kv_heads, head_dim, page, lengths, q_counts):
    from sprout_lm_b200 import kernels
    case = build_paged_case(dtype, heads, kv_heads, head_dim, page, lengths, q_counts)
    out = torch.empty(case["T"], heads * head_dim, dtype=dtype, device=DEV)
    kernels.attention_simple(case["q"], case["k_cache"], case["v_cache"], case["table"], case["seq_of_token"],
                             case["positions"], out, heads, kv_heads, head_dim, status)
    tol = 3e-6 if dtype == torch.float32 else 1.2e-2
    assert (out.double().cpu() - case["want"]).abs().max().item() <= tol
    assert int(status.item()) == 0


@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths,q_counts", [
    (14, 2, 64, 16, [300, 129, 16], [300, 1, 15]), (4, 4, 64, 8, [31, 32, 33], [31, 32, 33]), (2, 1, 128, 16, [128, 257, 1], [1, 130, 1]),
    (6, 2, 128, 4, [129], [127])])
def test_attention_tile(status, heads, kv_heads, head_dim, page, lengths, q_counts):
    """Edges of the 32-token tiles and the 128-key chunks, portions behind cached tokens: bit for bit the kernel of one token and
    head a block, also beside a value that only a later token sees and that is infinite."""
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.float32, heads, kv_heads, head_dim, page, lengths, q_counts)
    last = lengths[0] - 1                                         # the first request's last position
    case["v_cache"][case["table"][0, last // page].item(), :, last % page] = float("inf")
    one, tiled = torch.empty(case["T"], heads * head_dim, device=DEV), torch.empty(case["T"], heads * head_dim, device=DEV)
    kernels.attention_simple(case["q"], case["k_cache"], case["v_cache"], case["table"], case["seq_of_token"],
                             case["positions"], one, heads, kv_heads, head_dim, status)
    kernels.attention_tile(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"], case["positions"], tiled,
                           heads, kv_heads, head_dim, max(q_counts), status)
    assert torch.equal(one, tiled)
    assert torch.isfinite(tiled[:q_counts[0] - 1]).all() and torch.isinf(tiled[q_counts[0] - 1]).all()
    assert int(status.item()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("where", [0, 15, 16, 255, 256, 383, 500])
def test_attention_finds_one_far_key_among_hundreds(status, dtype, where):
    """The query equals one key scaled up: nearly all the weight lies on that key, at a page's
    first or last slot or far back; an attention that skips it returns something else."""
    from sprout_lm_b200 import kernels
    heads, kv_heads, head_dim, page = 4, 2, 32, 16
    case = build_paged_case(dtype, heads, kv_heads, head_dim, page, [40, 501], [1, 1], seed=where, spike=(1, where))
    out = torch.empty(case["T"], heads * head_dim, dtype=dtype, device=DEV)
    kernels.attention_simple(case["q"], case["k_cache"], case["v_cache"], case["table"], case["seq_of_token"],
                             case["positions"], out, heads, kv_heads, head_dim, status)
    tol = 3e-6 if dtype == torch.float32 else 1.5e-2
    assert (out.double().cpu() - case["want"]).abs().max().item() <= tol


DECODE_CASES = [
    (4, 2, 16, 16, [5, 17, 33, 1]), (3, 1, 32, 8, [61, 1, 130]), (14, 2, 64, 16, [300, 129, 16, 640, 513]),
    (5, 5, 48, 4, [40, 9]), (8, 2, 128, 16, [257, 64, 1000]), (6, 3, 80, 32, [100]), (16, 1, 256, 16, [70, 200]),
    (8, 2, 128, 16, [3000, 1200, 17]),                         # head size 128 through memory: swizzled rows, three CTAs per SM
    (6, 2, 96, 32, [2100, 5]),                                 # padded rows through memory
]


@pytest.mark.parametrize("split_keys", [None, 128, 256])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths", DECODE_CASES)
def test_attention_decode_split_keys(status, heads, kv_heads, head_dim, page, lengths, split_keys):
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * len(lengths))
    out = torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.attention_decode(case["q"], case["k_cache"], case["v_cache"], case["table"], case["context_lens"], out,
                             heads, kv_heads, head_dim, status, split_keys=split_keys)
    assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.2e-2
    # a wider block table (as under a captured graph) changes the split count, not the result
    wide = torch.full((len(lengths), case["table"].shape[1] + 19), -1, dtype=torch.int32, device=DEV)
    wide[:, :case["table"].shape[1]] = case["table"]
    again = torch.empty_like(out)
    kernels.attention_decode(case["q"], case["k_cache"], case["v_cache"], wide, case["context_lens"], again,
                             heads, kv_heads, head_dim, status, split_keys=split_keys)
    assert (again.double().cpu() - case["want"]).abs().max().item() <= 1.2e-2
    assert int(status.item()) == 0


@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths", DECODE_CASES[:6] + [
    (14, 2, 64, 16, [37 + 13 * i for i in range(70)]),        # a large batch: longer splits, few per request
    (4, 2, 64, 16, [6000, 1500]),                              # more than 8 splits: through memory too
    (4, 2, 64, 16, [2900 + 2 * i for i in range(80)]),         # more CTAs than four per SM: the variant held to five per SM's registers
    (6, 2, 32, 16, [5000 + 2 * i for i in range(60)]),
    (8, 2, 128, 16, [2500, 700, 90]),                          # head size 128 through memory
    (8, 4, 128, 32, [1300 + 7 * i for i in range(40)]),        # and with more CTAs than places
])
def test_attention_decode_fused_projection_tail(status, heads, kv_heads, head_dim, page, lengths, rotate):
    """The decode kernel that also finishes the projection: the new token's q, k, v arrive as
    float32 sums plus a bias; the kernel rotates, appends to the cache, attends and clears the sums.
    Compared with the separate rotary kernel followed by the decode kernel."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    R = len(lengths)
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * R, seed=3)
    width = (heads + 2 * kv_heads) * head_dim
    g = torch.Generator().manual_seed(11)
    sums = torch.randn(R, width, generator=g).to(DEV)
    bias = (torch.randn(width, generator=g) * 0.3).to(DEV)

    from sprout_lm_b200.parts import Runtime
    cos, sin = HalfSplitRotary("", head_dim, 1e4, max(1024, max(lengths))).rotary_tables(Runtime(DEV, torch.bfloat16)) if rotate else (None, None)
    positions = (case["context_lens"] - 1).to(torch.int32)
    seq_of_token = torch.arange(R, dtype=torch.int32, device=DEV)
    # the separate path
    k1, v1 = case["k_cache"].clone(), case["v_cache"].clone()
    acc1 = torch.zeros(R + 1, width, device=DEV)
    acc1[:R] = sums
    qkv = torch.zeros(R, width, dtype=torch.bfloat16, device=DEV)
    kernels.rope_append(qkv, positions, seq_of_token, case["table"], cos, sin, k1, v1, heads, kv_heads, head_dim, page,
                        True, status, acc=acc1[:R], bias=bias)
    want = torch.empty(R, heads * head_dim, dtype=torch.bfloat16, device=DEV)
    kernels.attention_decode(qkv[:, :heads * head_dim], k1, v1, case["table"], case["context_lens"], want, heads,
                             kv_heads, head_dim, status)
    # the fused kernel
    k2, v2 = case["k_cache"].clone(), case["v_cache"].clone()
    acc2 = sums.clone()
    got = torch.full_like(want, float("nan"))
    assert kernels.decode_fusable(R, heads, kv_heads, head_dim, case["table"].shape[1] * page)
    if max(lengths) > 5000:
        assert kernels.decode_split_plan(R, kv_heads, case["table"].shape[1] * page, head_dim)[2]      # this case goes through memory
    if R >= 60 and max(lengths) > 2000:
        _, splits, through_memory = kernels.decode_split_plan(R, kv_heads, case["table"].shape[1] * page, head_dim)
        assert through_memory and splits * kv_heads * R > 4 * kernels.sm_count()
    kernels.attention_decode_fused(acc2, bias, cos, sin, k2, v2, case["table"], case["context_lens"], got, heads,
                                   kv_heads, head_dim, status)
    assert torch.equal(k2, k1) and torch.equal(v2, v1)                 # the same append, bit for bit
    assert float(acc2.abs().max()) == 0.0                               # the sums are cleared
    assert (got.float() - want.float()).abs().max().item() <= 1.2e-2
    assert int(status.item()) == 0


RESIDENT_CASES = [
    (14, 2, 64, 16, [300, 129, 16, 640, 513, 1, 768, 32, 33]), (8, 2, 128, 16, [257, 64, 384, 1, 100]), (4, 4, 64, 8, [61, 1, 130, 8, 9]),
    (16, 1, 64, 128, [500, 128, 129]), (7, 1, 128, 32, [100, 31]), (3, 3, 64, 64, [64, 65, 700]),
]


@pytest.mark.parametrize("layout", ["scattered", "runs", "in order"])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths", RESIDENT_CASES)
def test_attention_decode_resident(status, heads, kv_heads, head_dim, page, lengths, fused, rotate, layout):
    """Decode attention with each request's whole context in one CTA's shared memory (pages by
    TMA; pages scattered, in runs, or in the pool's order): against the float64
    reference; in the fused form (sums in, rotation, cache append) also against the separate
    rotary kernel.  Every cache slot outside the requests is NaN."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts import Runtime
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    if rotate and not fused:
        pytest.skip("the rotation belongs to the fused form")
    R = len(lengths)
    room = kernels.decode_attention_plan(kernels.sm_count() // kv_heads, heads, kv_heads, head_dim, page, -(-max(lengths) // page) * page, max(lengths))
    assert room[0] == "resident"
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * R, seed=7, poison=True, layout=layout)
    out = torch.full((R, heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    if not fused:
        kernels.attention_decode_resident(case["k_cache"], case["v_cache"], case["table"], case["context_lens"], out, heads,
                                          kv_heads, head_dim, status, room[1], q=case["q"])
        assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.2e-2
        assert int(status.item()) == 0
        return
    width = (heads + 2 * kv_heads) * head_dim
    g = torch.Generator().manual_seed(11)
    sums = torch.randn(R, width, generator=g).to(DEV)
    bias = (torch.randn(width, generator=g) * 0.3).to(DEV)
    cos, sin = HalfSplitRotary("", head_dim, 1e4, 1024).rotary_tables(Runtime(DEV, torch.bfloat16)) if rotate else (None, None)
    positions = (case["context_lens"] - 1).to(torch.int32)
    seq_of_token = torch.arange(R, dtype=torch.int32, device=DEV)
    # the separate path on a cache without the poison beyond the requests (its kernels are tested for that elsewhere)
    clean = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * R, seed=7, layout=layout)
    k1, v1 = clean["k_cache"].clone(), clean["v_cache"].clone()
    acc1 = sums.clone()
    qkv = torch.zeros(R, width, dtype=torch.bfloat16, device=DEV)
    kernels.rope_append(qkv, positions, seq_of_token, case["table"], cos, sin, k1, v1, heads, kv_heads, head_dim, page,
                        True, status, acc=acc1, bias=bias)
    want = torch.empty(R, heads * head_dim, dtype=torch.bfloat16, device=DEV)
    kernels.attention_decode(qkv[:, :heads * head_dim], k1, v1, case["table"], case["context_lens"], want, heads,
                             kv_heads, head_dim, status, split_keys=128)
    k2, v2 = case["k_cache"].clone(), case["v_cache"].clone()
    acc2 = sums.clone()
    kernels.attention_decode_resident(k2, v2, case["table"], case["context_lens"], out, heads, kv_heads, head_dim, status,
                                      room[1], acc=acc2, bias=bias, cos_table=cos, sin_table=sin)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for r, n in enumerate(lengths):                         # the same append, bit for bit, and nothing else touched
        pg, slot = int(case["table"][r, (n - 1) // page]), (n - 1) % page
        assert torch.equal(k2[pg, :, slot], k1[pg, :, slot]) and torch.equal(v2[pg, :, slot], v1[pg, :, slot])
        k2[pg, :, slot] = case["k_cache"][pg, :, slot]
        v2[pg, :, slot] = case["v_cache"][pg, :, slot]
    same = lambda a, b: torch.equal(torch.nan_to_num(a.float(), nan=7.0), torch.nan_to_num(b.float(), nan=7.0))
    assert same(k2, case["k_cache"]) and same(v2, case["v_cache"])
    assert float(acc2.abs().max()) == 0.0                   # the sums are cleared
    assert (out.float() - want.float()).abs().max().item() <= 1.2e-2


@pytest.mark.parametrize("kernel", ["split", "resident"])
def test_decode_attention_applies_the_norms_scale_to_the_sums(status, kernel):
    """The fused decode kernels with ``norm_x``: the float32 sums are those of a product whose
    normalised input went without its scale; multiplied by 1 / rms of the request's row they must
    give what the same kernel gives for sums that were scaled beforehand."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts import Runtime
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    heads, kv_heads, head_dim, page = 14, 2, 64, 16
    lengths = [300, 129, 16, 640, 513, 1, 77, 33]
    R = len(lengths)
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * R, seed=9)
    width = (heads + 2 * kv_heads) * head_dim
    g = torch.Generator().manual_seed(13)
    sums = torch.randn(R, width, generator=g).to(DEV) * 3.0
    bias = (torch.randn(width, generator=g) * 0.3).to(DEV)
    x = (torch.randn(R, 200, generator=g) * torch.linspace(0.2, 4.0, R)[:, None]).to(DEV)     # rows of very different size
    eps = 1e-5
    inv = 1.0 / torch.sqrt((x.double() ** 2).mean(dim=1, keepdim=True) + eps)
    cos, sin = HalfSplitRotary("", head_dim, 1e4, 1024).rotary_tables(Runtime(DEV, torch.bfloat16))
    outs, caches = [], []
    for scaled_before in (True, False):
        acc = (sums.double() * inv).float() if scaled_before else sums.clone()
        k, v = case["k_cache"].clone(), case["v_cache"].clone()
        out = torch.empty(R, heads * head_dim, dtype=torch.bfloat16, device=DEV)
        norm_x = None if scaled_before else (x, eps)
        if kernel == "resident":
            kernels.attention_decode_resident(k, v, case["table"], case["context_lens"], out, heads, kv_heads, head_dim, status, 640,
                                              acc=acc, bias=bias, cos_table=cos, sin_table=sin, norm_x=norm_x)
        else:
            kernels.attention_decode_fused(acc, bias, cos, sin, k, v, case["table"], case["context_lens"], out, heads, kv_heads,
                                           head_dim, status, norm_x=norm_x)
        torch.cuda.synchronize()
        assert float(acc.abs().max()) == 0.0
        outs.append(out.float())
        caches.append((k.float(), v.float()))
    assert int(status.item()) == 0
    assert (outs[0] - outs[1]).abs().max().item() <= 2e-2                     # the scale in float32, before or inside: a bfloat16 step apart at most
    assert (caches[0][0] - caches[1][0]).abs().max().item() <= 4e-2 and (caches[0][1] - caches[1][1]).abs().max().item() <= 4e-2
    assert (outs[0].abs().max().item()) > 0.1


def test_attention_decode_resident_refuses_a_context_beyond_its_room(status):
    """A request longer than the launch has room for is flagged in the status word and gets no
    output; nothing is read or written out of bounds."""
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, 4, 2, 64, 16, [300, 40], [1, 1])
    out = torch.zeros(2, 4 * 64, dtype=torch.bfloat16, device=DEV)
    kernels.attention_decode_resident(case["k_cache"], case["v_cache"], case["table"], case["context_lens"], out, 4, 2, 64,
                                      status, 256, q=case["q"])
    torch.cuda.synchronize()
    assert int(status.item()) == 32
    status.zero_()
    assert float(out[0].float().abs().max()) == 0.0
    assert (out[1].double().cpu() - case["want"][1]).abs().max().item() <= 1.2e-2
    with pytest.raises(kernels.KernelError, match="cap_keys"):
        kernels.attention_decode_resident(case["k_cache"], case["v_cache"], case["table"], case["context_lens"], out, 4, 2, 64,
                                          status, 1024, q=case["q"])


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths", [(14, 2, 64, 16, [300, 129, 16, 640, 513, 1]),
                                                                   (3, 1, 48, 8, [61, 1, 130]), (4, 2, 64, 16, [3000, 70])])
def test_attention_decode_ignores_what_lies_beyond_a_request(status, heads, kv_heads, head_dim, page, lengths, fused):
    """Every cache slot that holds no key of a request is NaN: the rest of a last page (which the
    kernel's first pass loads before it knows the request's length), and pages nobody owns.  A
    page that another request used before holds whatever that request left; none of it may reach
    the result."""
    from sprout_lm_b200 import kernels
    R = len(lengths)
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, [1] * R, seed=5, poison=True)
    out = torch.full((R, heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    if not fused:
        kernels.attention_decode(case["q"], case["k_cache"], case["v_cache"], case["table"], case["context_lens"], out,
                                 heads, kv_heads, head_dim, status)
        assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.2e-2
    else:
        # the new token's q, k, v as sums: q is the case's query, k and v the case's last key and value
        width = (heads + 2 * kv_heads) * head_dim
        sums = torch.zeros(R, width, device=DEV)
        sums[:, :heads * head_dim] = case["q"].float()
        k, v = case["k_cache"].clone(), case["v_cache"].clone()
        for r, n in enumerate(lengths):
            pg, slot = int(case["table"][r, (n - 1) // page]), (n - 1) % page
            sums[r, heads * head_dim:(heads + kv_heads) * head_dim] = k[pg, :, slot].float().reshape(-1)
            sums[r, (heads + kv_heads) * head_dim:] = v[pg, :, slot].float().reshape(-1)
            k[pg, :, slot] = float("nan")                  # the kernel writes the new token's slot itself
            v[pg, :, slot] = float("nan")
        kernels.attention_decode_fused(sums, None, None, None, k, v, case["table"], case["context_lens"], out, heads,
                                       kv_heads, head_dim, status)
        assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.2e-2
        assert float(sums.abs().max()) == 0.0
    assert int(status.item()) == 0


@pytest.mark.parametrize("tokens,head_dim", [(3, 32), (20, 64)])
def test_rope_append_clears_the_sums_of_a_refused_position(status, tokens, head_dim):
    """A position beyond the rotary table is flagged and skipped; the float32 sums of that token
    must still be emptied, or the next product into the workspace would add to them."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.parts import Runtime
    from sprout_lm_b200.parts.rope import HalfSplitRotary
    heads, kv_heads, page = 4, 2, 16
    width = (heads + 2 * kv_heads) * head_dim
    cos, sin = HalfSplitRotary("", head_dim, 1e4, 64).rotary_tables(Runtime(DEV, torch.bfloat16))
    acc = rand(tokens, width, seed=2) + 3.0
    bias = rand(width, seed=3)
    positions = torch.arange(tokens, dtype=torch.int32, device=DEV)
    positions[1] = 64                                    # one past the table
    table = torch.arange(4, dtype=torch.int32, device=DEV).reshape(1, 4)
    k_cache = torch.zeros(4, kv_heads, page, head_dim, dtype=torch.bfloat16, device=DEV)
    v_cache = torch.zeros_like(k_cache)
    qkv = torch.zeros(tokens, width, dtype=torch.bfloat16, device=DEV)
    kernels.rope_append(qkv, positions, torch.zeros(tokens, dtype=torch.int32, device=DEV), table, cos, sin, k_cache,
                        v_cache, heads, kv_heads, head_dim, page, True, status, acc=acc, bias=bias)
    torch.cuda.synchronize()
    assert int(status.item()) == 16
    status.zero_()
    assert float(acc.abs().max()) == 0.0
    assert float(qkv[0].float().abs().max()) > 0 and float(qkv[1].float().abs().max()) == 0.0


def test_a_bounded_wait_runs_out_and_the_kernel_returns(status):
    """Every wait of the kernels on an mbarrier (a copy's arrival, a product's completion) is
    bounded in time.  A one-warp kernel waits, with that same helper, on a barrier on which nothing
    ever arrives: after the bound (about a second and a half) it gives up, sets the status word's
    wait bit and returns: no fault, no hang, and the device goes on working."""
    import time
    from sprout_lm_b200 import kernels
    torch.cuda.synchronize()
    begin = time.perf_counter()
    kernels.wait_probe(status)
    torch.cuda.synchronize()
    seconds = time.perf_counter() - begin
    assert int(status.item()) == 8 and kernels.describe_status(8) == "a bounded device-side wait ran out"
    assert 0.5 <= seconds <= 10.0, seconds
    status.zero_()
    out = torch.empty(2, 64, device=DEV)
    kernels.rmsnorm(torch.ones(2, 64, device=DEV), torch.ones(64, device=DEV), out, 1e-6)
    torch.cuda.synchronize()
    assert abs(float(out[0, 0]) - 1.0) < 1e-5 and int(status.item()) == 0


def test_sampling_never_draws_a_token_of_probability_zero(status):
    """A peaked row whose tail is far below: with the uniform number just under 1 the draw falls
    where rounding decides (the two kernels add the same exponentials in different orders); it must
    land on a token that has weight, not on the tail."""
    from sprout_lm_b200 import kernels
    vocab = 4099
    for heavy in (1, 5, 40):
        logits = torch.full((3, vocab), -1e30, device=DEV)
        logits[:, :heavy] = rand(3, heavy, scale=1.0, seed=heavy)
        logits[2, vocab - 1] = -80.0                              # a weight that underflows against the maximum
        out = torch.empty(3, dtype=torch.int32, device=DEV)
        temperature = torch.tensor([1.0, 0.7, 1.3], device=DEV)
        for u in (1.0 - 2.0 ** -24, 0.999, 0.5, 0.0):
            kernels.sample(logits, out, status, temperature, torch.full((3,), u, device=DEV))
            assert all(0 <= t < heavy for t in out.tolist()), (heavy, u, out.tolist())
    assert int(status.item()) == 0


@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths,q_counts", ATTN_CASES + [
    (14, 2, 64, 16, [700, 650, 2, 90], [700, 1, 2, 9]), (2, 1, 112, 8, [75], [75]), (7, 7, 96, 16, [33, 64], [2, 64])])
def test_attention_prefill_tensor_cores(status, heads, kv_heads, head_dim, page, lengths, q_counts):
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, q_counts)
    out = torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                              case["positions"], out, heads, kv_heads, head_dim, status)
    assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.5e-2
    assert int(status.item()) == 0


TC_PREFILL_CASES = [
    # heads, kv_heads, head_dim, page, cached lengths, queries of this step
    (14, 2, 64, 16, [700, 650, 2, 90], [700, 1, 2, 9]),       # several key tiles, rows of several requests
    (4, 2, 64, 8, [129, 128, 127], [129, 128, 1]),            # the edges of a key tile
    (8, 2, 128, 16, [300, 64], [37, 64]),                     # head_dim 128: two 64-element blocks, one P buffer
    (3, 1, 64, 32, [513], [200]),                             # a portion in the middle of a long request
    (2, 2, 128, 64, [260, 5], [260, 5]),
    (5, 1, 64, 128, [400], [400]),                            # a page as long as a key tile
    (2, 1, 64, 256, [600, 100], [90, 100]),                   # pages longer than a key tile
    (16, 1, 64, 16, [45], [45]),                              # many heads per key head: a tile holds few tokens
    (4, 1, 128, 128, [300, 129], [300, 70]),                  # head_dim 128 with pages of two key tiles
    (14, 2, 64, 16, [1500], [1500]),                          # Q tile 0 of a piece ends a key tile before Q tile 1
    (2, 2, 64, 16, [40, 128, 200], [40, 128, 129]),           # pieces with one Q tile and with two
]


@pytest.mark.parametrize("heads,kv_heads,head_dim,page,lengths,q_counts", TC_PREFILL_CASES)
def test_attention_prefill_tcgen05(status, heads, kv_heads, head_dim, page, lengths, q_counts):
    """The tcgen05 prefill kernel against the float64 reference, with NaN in every cache slot
    that holds no key: a kernel that lets one of them into a product shows it."""
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, lengths, q_counts, seed=5, poison=True)
    out = torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                              case["positions"], out, heads, kv_heads, head_dim, status, variant="tcgen05")
    assert int(status.item()) == 0
    err = (out.double().cpu() - case["want"]).abs().max(dim=1).values
    assert float(err.max()) <= 1.5e-2, f"token {int(err.argmax())} of {case['T']} differs by {float(err.max()):.3e}"
    # the other kernel on the same case (it must not read the poisoned slots either)
    again = torch.full_like(out, float("nan"))
    kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                              case["positions"], again, heads, kv_heads, head_dim, status, variant="mma_sync")
    assert float((again.double().cpu() - case["want"]).abs().max()) <= 1.5e-2


def test_attention_prefill_tcgen05_refuses_other_sizes(status):
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, 4, 2, 48, 16, [40], [40])
    out = torch.empty(case["T"], 4 * 48, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(kernels.KernelError, match="head_dim 64 or 128"):
        kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                                  case["positions"], out, 4, 2, 48, status, variant="tcgen05")


@pytest.mark.parametrize("where", [0, 127, 128, 255, 256, 700, 1023])
def test_tcgen05_prefill_finds_one_far_key(status, where):
    """One key among 1,024 whose score stands out, at the edges of the 128-key tiles."""
    from sprout_lm_b200 import kernels
    heads, kv_heads, head_dim, page = 4, 2, 64, 16
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, [1024], [40], seed=where, spike=(0, where))
    out = torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device=DEV)
    kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                              case["positions"], out, heads, kv_heads, head_dim, status, variant="tcgen05")
    assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.5e-2


@pytest.mark.parametrize("where", [0, 15, 16, 63, 64, 255, 256, 383, 500])
def test_fast_attention_finds_one_far_key(status, where):
    from sprout_lm_b200 import kernels
    heads, kv_heads, head_dim, page = 4, 2, 32, 16
    case = build_paged_case(torch.bfloat16, heads, kv_heads, head_dim, page, [40, 501], [1, 1], seed=where, spike=(1, where))
    for name in ("decode", "prefill"):
        out = torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device=DEV)
        if name == "decode":
            kernels.attention_decode(case["q"], case["k_cache"], case["v_cache"], case["table"], case["context_lens"],
                                     out, heads, kv_heads, head_dim, status)
        else:
            kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"],
                                      case["positions"], out, heads, kv_heads, head_dim, status)
        assert (out.double().cpu() - case["want"]).abs().max().item() <= 1.5e-2, name


# ------------------------------------------------------------------------------- sampling
@pytest.mark.parametrize("vocab", [7, 256, 509, 4099, 151936])
def test_sampling(status, vocab):
    from sprout_lm_b200 import kernels
    logits = rand(6, vocab, scale=2.0)
    logits[1, 3] = logits[1].max() + 1
    logits[1, vocab - 1] = logits[1, 3]                           # a tie: the lowest index wins
    out = torch.empty(6, dtype=torch.int32, device=DEV)
    kernels.sample(logits, out, status)
    assert out.tolist() == logits.argmax(-1).tolist() or out[1].item() == 3
    assert out[1].item() == 3
    temperature = torch.tensor([0.0, 0.8, 0.8, 1.5, 0.3, 0.8], device=DEV)
    for u in (0.0, 0.25, 0.5, 0.999999):
        uniform = torch.full((6,), u, device=DEV)
        kernels.sample(logits, out, status, temperature, uniform)
        assert out[0].item() == int(logits[0].argmax())
        for r in range(1, 6):
            p = torch.softmax(logits[r].double() / temperature[r].double(), 0)
            c = torch.cumsum(p, 0)
            pick = out[r].item()
            low = c[pick - 1].item() if pick else 0.0
            assert low - 1e-4 <= u <= c[pick].item() + 1e-4, (r, u, pick)
    assert int(status.item()) == 0
    logits[2, 1] = float("nan")
    kernels.sample(logits, out, status)
    assert out[2].item() == -1 and int(status.item()) & 4
    status.zero_()


# ------------------------------------------------------------------------------- attention with one or two maps on tcgen05
MAPS_CASES = [
    # maps, dim, vdim, heads, kv_heads, page, held, new, options
    (2, 64, 128, 8, 2, 16, [0], [300], dict(norm_eps=1e-5, lam=0.4)),
    (2, 64, 128, 4, 4, 16, [0, 513, 77], [129, 128, 385], dict(norm_eps=1e-5, lam=0.4, out_scale=0.5)),
    (2, 64, 64, 6, 2, 8, [40, 0], [100, 257], dict(lam=0.3, sink=True)),
    (1, 64, 128, 8, 2, 16, [700, 700, 0], [65, 200, 331], dict(mask=("window", 256), gate="head")),
    (1, 64, 128, 16, 4, 32, [1000, 37], [97, 640], dict(mask=("window", 300, 5), softcap=30.0)),
    (1, 64, 64, 14, 2, 16, [0, 0], [256, 1], dict()),
    (1, 64, 64, 7, 1, 64, [127, 128, 129], [128, 128, 255], dict(mask=("chunk", 200), sink=True)),
    (1, 128, 128, 4, 4, 16, [0, 300], [128, 700], dict(sink=True, softcap=20.0, gate="head")),
    (1, 128, 128, 8, 2, 128, [0], [1025], dict(mask=("chunk", 512), gate="element", turn="half")),
    (1, 64, 128, 4, 1, 16, [0], [2100], dict(mask=("window", 100), gate="element", turn="pairs", sink=True)),
    (1, 128, 128, 2, 1, 16, [5000], [130], dict()),
]


@pytest.mark.parametrize("divided", [False, True])
@pytest.mark.parametrize("maps,dim,vdim,heads,kv_heads,page,held,new,options", MAPS_CASES)
def test_maps_attention_tcgen05(status, monkeypatch, divided, maps, dim, vdim, heads, kv_heads, page, held, new, options):
    """The tcgen05 kernel against the float32-arithmetic kernel on the same bfloat16 inputs, with NaN in every cache slot that no
    query of the step sees and pages before a window given back; with and without a piece's keys divided among CTAs."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(dim + vdim + sum(new))
    total = [h + n for h, n in zip(held, new)]
    mask = options.get("mask")
    counts = [-(-t // page) for t in total]
    table = torch.full((len(new), max(counts) + 3), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(counts), generator=g).to(torch.int32), 0
    k = torch.full((sum(counts), kv_heads, page, maps * dim), float("nan"))
    v = torch.full((sum(counts), kv_heads, page, vdim), float("nan"))
    for r, t in enumerate(total):
        table[r, :counts[r]] = order[at:at + counts[r]]
        at += counts[r]
        first = 0 if mask is None else max(0, held[r] - mask[1] + 1) if mask[0] == "window" else held[r] // mask[1] * mask[1]
        keep = mask[2] if mask is not None and len(mask) > 2 else 0
        for pos in [*range(min(keep, first)), *range(first, t)]:
            k[table[r, pos // page], :, pos % page] = torch.randn(kv_heads, maps * dim, generator=g)
            v[table[r, pos // page], :, pos % page] = torch.randn(kv_heads, vdim, generator=g)
        for j in range(first // page):
            if j * page >= keep:
                table[r, j] = -1
    T = sum(new)
    dev = lambda x, dt=None: x.to(dt or x.dtype).to(DEV)
    starts = np.cumsum([0] + list(new))
    ctx = SimpleNamespace(
        seq_of_token=dev(torch.tensor([r for r, n in enumerate(new) for _ in range(n)], dtype=torch.int32)),
        positions=dev(torch.tensor([h + j for h, n in zip(held, new) for j in range(n)], dtype=torch.int32)),
        q_start=dev(torch.tensor(starts, dtype=torch.int32)), max_q_len=max(new), max_context=max(total), planned_context=0)
    cache = SimpleNamespace(k=dev(k, torch.bfloat16), v=dev(v, torch.bfloat16), block_table=dev(table), page_tokens=page)
    q = dev(torch.randn(T, heads * maps * dim, generator=g), torch.bfloat16)
    more = dict(mask=mask, softcap=options.get("softcap", 0.0))
    if options.get("sink"):
        more["sink"] = dev(torch.randn(heads, generator=g))
    if options.get("gate"):
        more["gate"] = dev(torch.randn(T, heads * (vdim if options["gate"] == "element" else 1), generator=g), torch.bfloat16)
    if options.get("turn"):
        angle = torch.rand(max(total), vdim // 2, generator=g) * 6.28
        more.update(turn=(dev(torch.cos(angle)), dev(torch.sin(angle))), interleaved=options["turn"] == "pairs")
    sizes = (heads, kv_heads, maps, dim, vdim, dim ** -0.5, options.get("lam", 0.0), options.get("norm_eps", 0.0), options.get("out_scale", 1.0), status)
    counters = torch.zeros(2 * kernels.sm_count(torch.device(DEV)), dtype=torch.int32, device=DEV) if divided else None
    got = torch.full((T, heads * vdim), float("nan"), dtype=torch.bfloat16, device=DEV)
    monkeypatch.setattr(kernels, "MAPS_TC_ROWS", 0)
    monkeypatch.setattr(kernels, "MAPS_TC_TILES", {})                # the kernel under test, whether it pays at these sizes or not
    kernels.multimap_attention(q, cache, ctx, got, *sizes, counters=counters, **more)
    assert int(status.item()) == 0
    assert counters is None or not counters.any()
    want = torch.empty(T, heads * vdim, dtype=torch.bfloat16, device=DEV)
    kernels.multimap_attention_simple(q, cache, ctx, want, *sizes, **more)
    status.zero_()                                 # the plain kernel flags the pages that were given back
    # probabilities rounded to 8 bits (2^-9 of each, of a sum whose terms are about as large as the result), the result rounded once
    # more on both sides; a norm over the head brings results to about one
    error = (got.float() - want.float())
    assert torch.isfinite(got).all()
    assert error.norm() <= 6e-3 * want.float().norm()
    assert error.abs().max() <= 4e-2 * want.float().abs().max()
    if divided:
        again = torch.empty_like(got)
        kernels.multimap_attention(q, cache, ctx, again, *sizes, counters=counters, **more)
        assert torch.equal(got, again) and not counters.any()


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("maps,dim,vdim,heads,kv_heads,page,options", [
    (1, 128, 128, 8, 2, 16, dict(softcap=30.0, sink=True, gate="head")), (1, 64, 128, 12, 1, 8, dict(mask=("window", 130, 5))),
    (1, 64, 64, 14, 2, 16, dict()), (1, 48, 48, 4, 4, 64, dict(mask=("chunk", 100), gate="element")), (1, 96, 96, 6, 2, 16, dict(turn="half")),
    (2, 64, 128, 8, 2, 16, dict(norm_eps=1e-5, lam=0.4)), (2, 128, 128, 4, 4, 32, dict(lam=0.3, sink=True)), (2, 16, 32, 16, 1, 8, dict(lam=0.3))])
def test_maps_attention_single_tokens(status, monkeypatch, whole, maps, dim, vdim, heads, kv_heads, page, options):
    """One token per request, contexts around a warp's 16 keys, a tile's 64 and the tiles that are on their way, with NaN in every slot
    that no query sees; a request's keys in one CTA or divided."""
    from sprout_lm_b200 import kernels
    if whole:
        monkeypatch.setattr(kernels, "multimap_key_split", lambda *a, **k: 1)
    held = [0, 1, 15, 16, 47, 63, 64, 127, 128, 191, 192, 255, 1300]
    test_maps_attention_tcgen05(status, monkeypatch, False, maps, dim, vdim, heads, kv_heads, page, held, [1] * len(held), options)


@pytest.mark.parametrize("maps,dim,vdim,mask,softcap", [(2, 64, 128, None, 0.0), (1, 64, 128, ("window", 700), 0.0), (1, 128, 128, None, 30.0), (1, 64, 64, None, 0.0)])
def test_maps_attention_tcgen05_is_as_close_to_64_bits(status, monkeypatch, maps, dim, vdim, mask, softcap):
    """A prompt's attention on tcgen05 is no further from float64 than on mma.sync: weights rounded relative to the row's own maximum, sums of
    weights in float32."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    heads, kv_heads, T, page, lam = 8, 2, 1536, 16, 0.4 if maps == 2 else 0.0
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + maps)
    make = lambda *shape: torch.randn(*shape, generator=g, device=DEV).to(torch.bfloat16)
    q, k, v = make(T, heads * maps * dim), make(T // page, kv_heads, page, maps * dim), make(T // page, kv_heads, page, vdim)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(seq_of_token=ints([0] * T), positions=ints(list(range(T))), q_start=ints([0, T]), max_q_len=T, max_context=T, planned_context=0)
    cache = SimpleNamespace(k=k, v=v, block_table=ints([list(range(T // page))]), page_tokens=page)
    at = torch.arange(T, device=DEV)
    hidden = at[None] > at[:, None]
    if mask is not None:
        hidden |= at[None] <= at[:, None] - mask[1]
    want = torch.zeros(T, heads, vdim, dtype=torch.float64, device=DEV)
    for h in range(heads):
        kh, vh = (x[:, h // (heads // kv_heads)].reshape(T, -1).double() for x in (k, v))
        for m in range(maps):
            part = slice(m * dim, (m + 1) * dim)
            score = q.view(T, heads, maps * dim)[:, h, part].double() @ kh[:, part].T * dim ** -0.5
            score = softcap * torch.tanh(score / softcap) if softcap else score
            want[:, h] += (1.0 if m == 0 else -lam) * (torch.softmax(score.masked_fill(hidden, -math.inf), -1) @ vh)
    error = {}
    for choice in ("mma_sync", "auto"):
        monkeypatch.setenv("SPROUT_MULTIMAP_ATTENTION", choice)
        out = torch.empty(T, heads * vdim, dtype=torch.bfloat16, device=DEV)
        kernels.multimap_attention(q, cache, ctx, out, heads, kv_heads, maps, dim, vdim, dim ** -0.5, lam, 0.0, 1.0, status, mask=mask, softcap=softcap)
        error[choice] = float((out.double().view(want.shape) - want).norm() / want.norm())
    assert int(status.item()) == 0 and 0 < error["auto"] < 5e-3
    # the two errors are norms over more than 700,000 roundings each: equal ones differ by a few thousandths
    assert error["auto"] <= 1.005 * error["mma_sync"], error


@pytest.mark.parametrize("maps,dim,vdim,rot,options", [
    (2, 64, 128, 64, {}), (1, 128, 128, 32, dict(weights=True)), (1, 64, 128, 64, dict(unit=True, turn=True)), (1, 32, 64, 16, dict(growth=True)),
    (2, 16, 32, 0, dict(growth=True, unit=True)), (1, 128, 128, 128, dict(interleaved=True, turn=True, weights=True)), (1, 128, 128, 64, dict(from_key=True, unit=True)),
    (1, 64, 64, 64, dict(read_only=True)), (1, 64, 24, 0, {})])
def test_rope_maps_append_in_16_byte_accesses(status, maps, dim, vdim, rot, options):
    """The 16-byte form against the general one (rows that do not start on 16 bytes take that one), with a page that is missing."""
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(dim + vdim + rot)
    heads, kv_heads, page, T = 6, 2, 4, 37
    write = not options.get("read_only")
    widths = [heads * maps * dim, kv_heads * maps * dim if write else 0, 0 if options.get("from_key") or not write else kv_heads * vdim]
    dev = lambda x, dt=None: x.to(dt or x.dtype).to(DEV)
    plain = torch.randn(T, sum(widths), generator=g).to(torch.bfloat16)
    positions, seqs = dev(torch.arange(T, dtype=torch.int32)), dev(torch.zeros(T, dtype=torch.int32))
    table = torch.randperm(12, generator=g).to(torch.int32)[None]
    table[0, 5] = -1
    table = dev(table)
    angle = torch.rand(64, max(rot, 2) // 2, generator=g) * 6.28
    cos, sin = (dev(torch.cos(angle)), dev(torch.sin(angle))) if rot else (None, None)
    more = dict(unit_eps=1e-5 if options.get("unit") else 0.0, value_from_key=bool(options.get("from_key")), interleaved=bool(options.get("interleaved")))
    if options.get("weights"):
        more.update(q_weight=dev(torch.randn(dim, generator=g)), k_weight=dev(torch.randn(dim, generator=g)), weight_eps=1e-5)
    if options.get("growth"):
        more["growth"] = (0.3, 7)
    if options.get("turn"):
        angle = torch.rand(64, vdim // 2, generator=g) * 6.28
        more["value_turn"] = (dev(torch.cos(angle)), dev(torch.sin(angle)))
    results = []
    for extra in (0, 1):                                    # rows of 8 elements and more, or of an odd number
        rows = torch.zeros(T, -(-sum(widths) // 8) * 8 + extra, dtype=torch.bfloat16, device=DEV)
        rows[:, :sum(widths)] = plain.to(DEV)
        k = torch.zeros(12, kv_heads, page, maps * dim, dtype=torch.bfloat16, device=DEV)
        v = torch.zeros(12, kv_heads, page, vdim, dtype=torch.bfloat16, device=DEV)
        status.zero_()
        kernels.rope_maps_append(rows, positions, seqs, table, cos, sin, k if write else None, v if write else None, heads * maps, kv_heads, maps, dim, vdim, page,
                                 write, status, **more)
        results.append((rows[:, :sum(widths)].float(), k.float(), v.float(), int(status.item())))
    status.zero_()
    assert results[0][3] == results[1][3] == (1 if write else 0)
    for fast, general in zip(results[0][:3], results[1][:3]):
        # one rounding to bfloat16 of float32 results whose sums are added in another order
        assert ((fast - general).abs() <= 2 ** -7 * general.abs() + 1e-6).all()


@pytest.mark.parametrize("unit", ["clamped_glu", "plain", "silu_glu"])
@pytest.mark.parametrize("counts,width,ff,weighted", [([256, 0, 257, 1, 1540], 512, 256, False), ([0, 2050, 0, 3], 520, 264, True), ([17] * 40, 1032, 1040, True)])
def test_experts_on_tcgen05(status, monkeypatch, unit, counts, width, ff, weighted):
    """Experts without rows, with one, at the edges of the 256-row tiles, sizes that no tile divides: against the CUDA-core products."""
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(width + ff)
    experts, entries, top = len(counts), sum(counts), 1
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(entries, generator=g)].to(torch.int32)[:, None].to(DEV)
    offsets, order = torch.zeros(experts + 1, dtype=torch.int32, device=DEV), torch.zeros(entries, dtype=torch.int32, device=DEV)
    place = torch.zeros(entries, dtype=torch.int32, device=DEV)
    kernels.moe_arrange(ids, torch.tensor(counts, dtype=torch.int32, device=DEV), offsets, order, place, experts)
    make = lambda *shape, scale=1.0: (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).to(DEV)
    h = make(entries, width)
    w_up, w_down = make(experts, (1 if unit == "plain" else 2) * ff, width, scale=width ** -0.5), make(experts, width, ff, scale=ff ** -0.5)
    weights = torch.rand(entries, 1, generator=g).to(DEV) if weighted else None
    limit = 7.0 if unit == "clamped_glu" else 0.0
    results = []
    monkeypatch.setattr(kernels, "EXPERTS_TC_ELEMENTS", 0)           # the kernel under test, whether it pays at these sizes or not
    for choice in ("mma", "plain"):
        monkeypatch.setenv("SPROUT_MOE", choice)
        act = torch.zeros(entries, ff, dtype=torch.bfloat16, device=DEV)
        rows = torch.zeros(entries, width, device=DEV)
        kernels.moe_experts(h, order, offsets, w_up, w_down, act, rows, experts, top, limit, 1.702, unit=unit, row_weights=weights, status=status)
        results.append((act.float(), rows))
    assert kernels.load_library().sprout_moe_tc_supported(entries, experts, top, width, ff, width) and int(status.item()) == 0
    # float32 sums in another order; a product on the edge of a bfloat16 rounding moves its activation by 2^-8 of itself
    for tc, plain in zip(*results):
        assert (tc - plain).norm() <= 2 ** -9 * plain.norm()
        assert (tc - plain).abs().max() <= 2 ** -6 * plain.abs().max()


@pytest.mark.parametrize("tokens,hidden,ff,stride", [(1, 512, 256, 512), (257, 520, 328, 1040), (700, 1032, 1040, 1032)])
def test_clamped_glu_product(status, monkeypatch, tokens, hidden, ff, stride):
    """A gated unit's product with the activation in its epilogue against the product and the activation's kernel, rows side by side or apart."""
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(tokens)
    h = torch.randn(tokens, stride, generator=g).to(torch.bfloat16).to(DEV)[:, :hidden]
    w = (torch.randn(2 * ff, hidden, generator=g) * 2.0 * hidden ** -0.5).to(torch.bfloat16).to(DEV)
    got, want = (torch.zeros(tokens, ff, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    monkeypatch.setattr(kernels, "GLU_PRODUCT_TILES", 0)             # the kernel under test, whether it pays at these sizes or not
    assert kernels.clamped_glu_product(h, w, got, 2.0, 1.702, status) and int(status.item()) == 0
    gate_up = torch.empty(tokens, 2 * ff, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_bf16(h, w, gate_up, status)
    kernels.glu_clamped(gate_up, want, 2.0, 1.702)
    # a product on the edge of a bfloat16 rounding moves its activation by 2^-8 of itself
    error = got.float() - want.float()
    assert error.norm() <= 2 ** -9 * want.float().norm() and error.abs().max() <= 2 ** -6 * want.float().abs().max()


@pytest.mark.parametrize("unit", ["clamped_glu", "silu_glu", "dense"])
def test_gated_units_of_exact_products(status, monkeypatch, unit):
    """The same activation in every kernel, bit for bit, where the products are exact (a matrix of ones and zeros picks them), for gates whose exponential is
    nothing, everything and nearly too large for float32."""
    from sprout_lm_b200 import kernels
    tokens, ff = 600, 256
    h = torch.cat([torch.linspace(-92.0, 30.0, tokens * ff).view(tokens, ff), torch.linspace(-9.0, 9.0, tokens * ff).view(ff, tokens).T], 1)
    special = torch.tensor([0.0, 1e-38, -1e-38, 3e38, -3e38, -89.0, -300.0])
    h[0, :len(special)] = special
    h = h.to(torch.bfloat16).to(DEV)
    w = torch.eye(2 * ff, dtype=torch.bfloat16, device=DEV)
    if unit == "dense":
        monkeypatch.setattr(kernels, "GLU_PRODUCT_TILES", 0)
        got, want = (torch.zeros(tokens, ff, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        assert kernels.clamped_glu_product(h, w, got, 7.0, 1.0, status)
        kernels.glu_clamped(h, want, 7.0, 1.0)
        results = [got, want]
    else:
        order, offsets = torch.arange(tokens, dtype=torch.int32, device=DEV), torch.tensor([0, tokens], dtype=torch.int32, device=DEV)
        down, results = torch.zeros(1, 2 * ff, ff, dtype=torch.bfloat16, device=DEV), []
        monkeypatch.setattr(kernels, "EXPERTS_TC_ELEMENTS", 0)
        for choice in ("mma", "mma_sync", "plain"):
            monkeypatch.setenv("SPROUT_MOE", choice)
            act = torch.zeros(tokens, ff, dtype=torch.bfloat16, device=DEV)
            kernels.moe_experts(h, order, offsets, w[None], down, act, torch.zeros(tokens, 2 * ff, device=DEV), 1, 1, 7.0 if unit == "clamped_glu" else 0.0, 1.0,
                                unit=unit, status=status)
            results.append(act)
    assert int(status.item()) == 0
    for other in results[1:]:
        assert torch.equal(results[0].view(torch.int16), other.view(torch.int16))


@pytest.mark.parametrize("tokens,weighted", [(1, False), (2, True), (3, False), (40, True)])
def test_routed_in_one_call(status, tokens, weighted):
    """Router, arrangement and products behind one call (a few tokens on the few-token kernel, more on tcgen05) give what they give one after another, bit for bit."""
    from sprout_lm_b200 import kernels
    experts, top, width, ff = 8, 2, 512, 512
    g = torch.Generator().manual_seed(tokens)
    make = lambda *shape: (torch.randn(*shape, generator=g) * shape[-1] ** -0.5).to(torch.bfloat16).to(DEV)
    h, w_up, w_down, router = make(tokens, width), make(experts, 2 * ff, width), make(experts, width, ff), torch.randn(experts, width, generator=g).to(DEV)
    counts, offsets = torch.zeros(experts, dtype=torch.int32, device=DEV), torch.zeros(experts + 1, dtype=torch.int32, device=DEV)
    got_ids, got_weights, got_place, got_rows = kernels.moe_routed(h, router, None, counts, offsets, w_up, w_down, experts, top, 1.5, 7.0, 1.7,
                                                                   unit="clamped_glu", weight_on_input=weighted, status=status)
    ids, weights = torch.zeros(tokens, top, dtype=torch.int32, device=DEV), torch.zeros(tokens, top, device=DEV)
    order, place = (torch.zeros(tokens * top, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_route(h, router, None, ids, weights, counts, experts, top, 1.5)
    kernels.moe_arrange(ids, counts, offsets, order, place, experts)
    act, rows = torch.empty(tokens * top, ff, dtype=torch.bfloat16, device=DEV), torch.empty(tokens * top, width, device=DEV)
    kernels.moe_experts(h, order, offsets, w_up, w_down, act, rows, experts, top, 7.0, 1.7, unit="clamped_glu", row_weights=weights if weighted else None, status=status)
    assert torch.equal(got_ids, ids) and torch.equal(got_weights, weights) and int(status.item()) == 0
    # entries of an expert may lie in another order: an entry's row is compared
    assert torch.equal(got_rows[got_place.flatten().long()], rows[place.long()])


@pytest.mark.parametrize("unit", ["clamped_glu", "plain"])
def test_experts_tiles_of_every_width(status, monkeypatch, unit):
    """Rows of an expert in one tile of 16 to 256 columns, in two and more of equal size, features and K that no tile divides."""
    test_experts_on_tcgen05(status, monkeypatch, unit, [15, 16, 31, 33, 240, 241, 255, 513, 0, 783, 4353], 648, 328, False)


@pytest.mark.parametrize("experts,entries", [(1, 1), (5, 1025), (32, 9000), (33, 8193), (1025, 9000), (2048, 700)])
def test_entries_arranged_by_expert(experts, entries):
    """Offsets from the counts, every entry once within its expert, identity experts without a place, the counts left zeroed."""
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(experts + entries)
    ids = torch.randint(0, experts + 2, (entries, 1), generator=g).to(torch.int32)      # the last two: identity experts
    counts = torch.bincount(ids.flatten().long(), minlength=experts + 2)[:experts]
    device_counts = counts.to(torch.int32).to(DEV)
    offsets, order = torch.zeros(experts + 1, dtype=torch.int32, device=DEV), torch.zeros(entries, dtype=torch.int32, device=DEV)
    place = torch.zeros(entries, dtype=torch.int32, device=DEV)
    kernels.moe_arrange(ids.to(DEV), device_counts, offsets, order, place, experts)
    want = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    total = int(want[-1])
    order, place = order.cpu().long()[:total], place.cpu().long()
    assert (offsets.cpu().long() == want).all() and (device_counts == 0).all()
    assert (order.sort().values == torch.nonzero(ids.flatten() < experts).flatten()).all()
    assert (ids.flatten().long()[order] == torch.repeat_interleave(torch.arange(experts), counts)).all()
    assert (place[order] == torch.arange(total)).all() and (place[ids.flatten() >= experts] == -1).all()


@pytest.mark.parametrize("window,sink,interleaved,dim,tail,vdim", [(None, True, True, 64, 64, 128), (100, False, False, 64, 64, 128), (64, True, True, 64, 0, 64), (None, True, False, 64, 64, 128)])
@pytest.mark.parametrize("held,new", [([0], [129]), ([0, 300, 65], [400, 129, 190])])
def test_latent_attention_unfolded(monkeypatch, window, sink, interleaved, dim, tail, vdim, held, new):
    """A latent attention layer's unfolded form against its folded form, portions behind cached rows, pages before a window given back."""
    from sprout_lm_b200 import kernels
    from sprout_lm_b200.config.specs import PartSpec
    from sprout_lm_b200.engine.batch import StepContext
    from sprout_lm_b200.parts import CacheView, Runtime, WeightSource, build_part
    g = torch.Generator().manual_seed(sum(new) + dim + tail)
    heads, rank, width, page = 4, 128, 256, 16
    position = PartSpec("none", {}) if not tail else PartSpec("rope_interleaved" if interleaved else "rope_yarn", {"dims": tail, "theta": 1e4, "max_positions": 1024})
    part = build_part("mixer", PartSpec("latent_attention", dict(hidden_size=width, heads=heads, dim=dim, rot_dim=tail, value_dim=vdim, kv_rank=rank, q_rank=64,
                                                                 scale=0.1, eps=1e-5, position=position, sink=sink, window=window)))
    decls = {d.name: d for d in part.tensor_decls()}
    weights = {name: torch.randn(d.shape, generator=g) * d.shape[-1] ** -0.5 + (d.init == "gain") for name, d in decls.items()}
    part.load(WeightSource(lambda name: weights[name], Runtime(DEV, torch.bfloat16)))
    total = [h + n for h, n in zip(held, new)]
    counts = [-(-t // page) for t in total]
    pages = torch.randperm(sum(counts), generator=g).to(torch.int32)
    table, at = torch.full((len(new), 64), -1, dtype=torch.int32), 0
    cache = torch.randn(sum(counts), 1, page, rank + tail, generator=g)
    for r in range(len(new)):
        table[r, :counts[r]] = pages[at:at + counts[r]]
        at += counts[r]
        for j in range(max(0, held[r] - (window or 10 ** 6) + 1) // page):
            cache[table[r, j]] = float("nan")
            table[r, j] = -1
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
    starts = np.cumsum([0] + new).tolist()
    T = sum(new)
    ctx = StepContext(num_tokens=T, num_seqs=len(new), max_q_len=max(new), max_context=max(total), token_ids=ints([0] * T),
                      positions=ints([h + j for h, n in zip(held, new) for j in range(n)]), seq_of_token=ints([i for i, n in enumerate(new) for _ in range(n)]),
                      q_start=ints(starts), context_lens=ints(total), state_slots=ints([0] * len(new)), logits_rows=ints([0]), block_tables=[table.to(DEV)], page_tokens=page)
    h = torch.randn(T, width, generator=g).to(torch.bfloat16).to(DEV)
    results = []
    monkeypatch.setattr(kernels, "UNFOLD_STEP", 128)
    monkeypatch.setattr(kernels, "UNFOLD_GAIN", 1e9)                 # the form under test, whether it pays at these sizes or not
    for rows in (kernels.UNFOLD_ROWS, 0):
        monkeypatch.setattr(kernels, "UNFOLD_ROWS", rows)
        view = CacheView(cache.to(torch.bfloat16).to(DEV), None, ctx.block_tables[0], page, True)
        assert bool(kernels.latent_unfold_rows(ctx, view, T, heads, dim, tail, vdim, rank, tail, window or 0)) == bool(rows)
        x = torch.zeros(T, width, device=DEV)
        part.forward(h, x, ctx, view)
        assert int(part.runtime.status.item()) == 0 and torch.isfinite(x).all()
        results.append(x)
    # two forms of the same sums with the intermediate results rounded to bfloat16 at other places
    assert (results[0] - results[1]).norm() <= 1.5e-2 * results[1].norm()


@pytest.mark.parametrize("rows,part,groups,period,gate_dtype,gate_first,silu", [
    (1, 4, 1, 4, None, False, True), (7, 64, 6, 64, torch.float32, True, True), (33, 100, 3, 300, torch.bfloat16, False, False),
    (5, 128, 9, 128, torch.bfloat16, True, False), (3, 136, 5, 680, torch.float32, False, True), (70, 256, 2, 256, torch.bfloat16, False, True),
    # from 1,024 parts on a group of lanes has a part, below a block
    (1023, 4, 1, 4, None, False, True), (1025, 4, 1, 4, None, False, True), (171, 64, 6, 64, torch.float32, True, True),
    (343, 100, 3, 300, torch.bfloat16, False, False), (114, 128, 9, 128, torch.bfloat16, True, False), (205, 136, 5, 680, torch.float32, False, True),
    (513, 256, 2, 256, torch.bfloat16, False, True),
    # around the sizes at which a lane takes eight elements, and beyond what a warp's lanes hold in fours
    *[(rows, part, groups, part * (groups if wide else 1), gate, first, silu) for rows, groups in ((343, 3), (340, 3), (1024, 1))
      for part, wide, gate, first, silu in ((60, True, None, False, True), (68, False, torch.bfloat16, False, True), (124, True, torch.float32, True, False),
                                            (132, False, None, False, True), (132, True, torch.bfloat16, True, True), (252, True, torch.bfloat16, False, False))]])
def test_gated_group_norm_lanes(rows, part, groups, period, gate_dtype, gate_first, silu):
    """A part per group of lanes: the smallest and largest parts, lanes without elements, a last warp that is not full, every kind of gate."""
    from sprout_lm_b200 import kernels
    g = torch.Generator().manual_seed(rows + part)
    width = part * groups
    o = torch.randn(rows, width, generator=g)
    weight = torch.randn(period, generator=g)
    wide = torch.randn(rows, width + 16, generator=g)
    gate = None if gate_dtype is None else wide.to(gate_dtype)
    out = torch.full((rows, width), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gated_group_norm(o.to(DEV), None if gate is None else gate.to(DEV)[:, :width], weight.to(DEV), out, 1e-5, groups, gate_first, silu)
    factor = torch.ones(rows, width, dtype=torch.float64)
    if gate is not None:
        z = gate[:, :width].double()
        factor = torch.sigmoid(z) * (z if silu else 1.0)
    v = (o.double() * (factor if gate_first else 1.0)).view(rows, groups, part)
    want = ((v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5)).view(rows, width) * weight.double().repeat(width // period)) * (1.0 if gate_first else factor)
    # one rounding to bfloat16 (2^-9 of the result) and a few float32 operations
    assert ((out.double().cpu() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("outputs,extra,width", [(32, 0, 1024), (37, 1, 520), (37, 1, 516), (34, 0, 517), (15, 1, 40), (70, 2, 260)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_of_many_tokens(dtype, outputs, extra, width):
    """A step of many tokens (an output a warp or four, by the outputs and the type) picks and weighs as steps of a few tokens do, bit for bit: a
    token's sums have one order in all forms."""
    from sprout_lm_b200 import kernels
    T, top, g = 333, 4, torch.Generator().manual_seed(outputs)
    h = torch.randn(T, width, generator=g).to(dtype).to(DEV)
    router = (torch.randn(outputs + extra, width, generator=g) * width ** -0.5).to(DEV)
    correction = (torch.randn(outputs, generator=g) * 0.1).to(DEV)

    def route(rows):
        n = rows.shape[0]
        ids, weights = torch.zeros(n, top, dtype=torch.int32, device=DEV), torch.zeros(n, top, device=DEV)
        counts, more = torch.zeros(outputs, dtype=torch.int32, device=DEV), torch.zeros(n, extra, device=DEV) if extra else None
        kernels.moe_route(rows, router, correction, ids, weights, counts, outputs, top, 2.5, extra_out=more)
        return ids, weights, counts, more
    whole, parts = route(h), [route(h[i:i + 9].contiguous()) for i in range(0, T, 9)]
    assert torch.equal(whole[0], torch.cat([p[0] for p in parts])) and torch.equal(whole[2], sum(p[2] for p in parts))
    assert torch.equal(whole[1], torch.cat([p[1] for p in parts]))
    if extra:
        assert torch.equal(whole[3], torch.cat([p[3] for p in parts]))


def scan_oracle(form, q, k, v, decay, factor, extra, state):
    """The gated scan of one request in float64, all heads at once: q [n, H, dim], k likewise, v [n, H, vdim], decay [n, H, dim], factor [n, H] on k;
    ``extra``: the bonus [H, dim].  ``state`` [H, dim, vdim] is brought up to date; returns o [n, H, vdim]."""
    out = np.zeros(v.shape)
    for t in range(q.shape[0]):
        write = (1.0 - decay[t]) if form == "floor" else k[t] * factor[t][:, None]
        own = write[:, :, None] * v[t][:, None, :]
        before = state.copy() if form == "bonus" else None
        state *= decay[t][:, :, None]
        state += own
        seen = state if before is None else before + extra[:, :, None] * own
        out[t] = np.einsum("hdv,hd->hv", seen, q[t])
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", ["channel", "head", "floor", "bonus", "given"])
@pytest.mark.parametrize("dim,vdim", [(8, 600), (16, 24), (32, 130), (64, 37), (128, 33), (256, 16), (256, 21)])
def test_gated_scan_rows_in_16_byte_fetches(status, dtype, form, dim, vdim):
    """Chunked walks at every key size that fills the tile's slices (a batch then has 2 to 8 tokens and 16 to 512 columns a block, and at 256
    fewer values than the block has threads), in every form of decay: outputs and states against the recurrence in float64."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    heads, lengths, slots = 2, [131, 1, 66], [2, 0, 3]
    g = torch.Generator().manual_seed(dim + vdim)
    T, v_cols = sum(lengths), vdim - 3 if form == "given" else vdim
    make = lambda *shape: torch.randn(*shape, generator=g).to(dtype)
    q, k, v = make(T, heads * dim), make(T, heads * dim), make(T, heads * v_cols)
    z = 2.0 * torch.randn(T, heads if form in ("head", "given") else heads * dim, generator=g)
    z = z.to(dtype)
    bias = torch.linspace(-2.0, 1.0, heads) if form == "head" else torch.linspace(-3.0, 3.0, heads * dim)
    a_log = torch.linspace(-4.0, 0.3, heads)
    floor, bonus = torch.linspace(0.05, 0.98, heads * dim), torch.linspace(-1.0, 1.5, heads * dim)
    tau, scale = 3.0, 0.5
    f64 = lambda t: t.double().numpy()
    sigmoid = lambda x: 1.0 / (1.0 + np.exp(-x))
    factor = np.ones((T, heads))
    more = {}
    if form == "given":
        given = torch.rand(T, heads, generator=g), torch.rand(T, heads, generator=g)
        decay, factor = np.repeat(f64(given[0])[:, :, None], dim, axis=2), f64(given[1])
        more = dict(given=tuple(t.to(DEV) for t in given), ones_col=True)
    elif form == "head":
        factor = np.logaddexp(0.0, f64(z) + f64(bias))
        decay = np.repeat(np.exp(-np.exp(f64(a_log)) * factor)[:, :, None], dim, axis=2)
        more = dict(per_head=True, a_log=a_log.to(DEV))
    else:
        x = (f64(z) + f64(bias)).reshape(T, heads, dim)
        if form == "channel":
            decay, more = sigmoid(x) ** (1.0 / tau), dict(tau=tau)
        elif form == "floor":
            low = f64(floor).reshape(heads, dim)
            decay, more = low + (1.0 - low) * sigmoid(x), dict(floor=floor.to(DEV))
        else:
            decay, more = np.exp(-np.exp(x)), dict(bonus=bonus.to(DEV))
    start = torch.randn(5, heads, dim, vdim, generator=g)
    want, want_state, at = np.zeros((T, heads, vdim)), f64(start).copy(), 0
    rows = lambda t, width: f64(t).reshape(T, heads, width)
    values = rows(v, v_cols)
    if form == "given":
        values = np.concatenate([values, np.ones((T, heads, 1)), np.zeros((T, heads, 2))], axis=2)
    for n, slot in zip(lengths, slots):
        part = slice(at, at + n)
        want[part] = scan_oracle(form, rows(q, dim)[part] * scale, rows(k, dim)[part], values[part], decay[part], factor[part],
                                 f64(bonus).reshape(heads, dim), want_state[slot])
        at += n
    ctx = SimpleNamespace(q_start=torch.tensor(np.cumsum([0] + lengths), dtype=torch.int32, device=DEV), max_q_len=max(lengths))
    state = SimpleNamespace(buffer=start.to(DEV), slots=torch.tensor(slots, dtype=torch.int32, device=DEV))
    out = torch.full((T, heads * vdim), float("nan"), device=DEV)
    kernels.gated_scan(q.to(DEV), None if form == "floor" else k.to(DEV), v.to(DEV), None if form == "given" else z.to(DEV),
                       None if form == "given" else bias.to(DEV), ctx, state, out, heads, heads, dim, vdim, status, q_scale=scale, **more)
    assert int(status.item()) == 0
    # float32 recurrences of up to 131 steps and sums over up to 256 products of terms of both signs: some 400 roundings of 2^-24
    for got, expected in ((out.double().cpu().numpy().reshape(want.shape), want), (state.buffer.double().cpu().numpy(), want_state)):
        assert np.abs(got - expected).max() <= 2.5e-5 * max(1.0, np.abs(expected).max())


@pytest.mark.parametrize("form", ["channel", "head", "given"])
@pytest.mark.parametrize("strength", [0.02, 1.0, 60.0])
@pytest.mark.parametrize("dim,vdim,ones", [(64, 8, False), (64, 72, False), (128, 64, False), (128, 136, False), (128, 130, True), (64, 65, True)])
def test_gated_scan_16_tokens_at_a_time(status, form, strength, dim, vdim, ones):
    """The walk on tensor cores: portions that end within 16 tokens and within a chunk, a single token, value columns short of a block's and beyond one,
    the column of ones, heads that share their keys, decays from almost none to all at once; outputs and states against the recurrence in float64."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    heads, groups, lengths, slots = 4, 2, [145, 1, 66, 128, 17], [2, 0, 3, 5, 1]
    g = torch.Generator().manual_seed(dim + vdim)
    T, v_cols = sum(lengths), vdim // 8 * 8
    make = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
    q, k, v = make(T, groups * dim), make(T, groups * dim), make(T, heads * v_cols)
    f64 = lambda t: t.double().numpy()
    factor, skip = np.ones((T, heads)), torch.linspace(-1.0, 1.0, heads)
    z = bias = None
    if form == "given":
        given = (torch.rand(T, heads, generator=g) ** strength, torch.rand(T, heads, generator=g))
        decay, factor = np.repeat(f64(given[0])[:, :, None], dim, axis=2), f64(given[1])
        more = dict(given=tuple(t.to(DEV) for t in given))
    elif form == "head":
        z, bias, a_log = torch.randn(T, heads, generator=g), torch.linspace(-2.0, 1.0, heads), torch.full((heads,), math.log(strength))
        factor = np.logaddexp(0.0, f64(z) + f64(bias))
        decay = np.repeat(np.exp(-strength * factor)[:, :, None], dim, axis=2)
        more = dict(per_head=True, a_log=a_log.to(DEV))
    else:
        z, bias = 2.0 * torch.randn(T, heads * dim, generator=g), torch.linspace(-3.0, 3.0, heads * dim)
        x = (f64(z) + f64(bias)).reshape(T, heads, dim)
        decay, more = (1.0 / (1.0 + np.exp(-x))) ** strength, dict(tau=1.0 / strength)
    start = torch.randn(7, heads, dim, vdim, generator=g)
    want, want_state, at = np.zeros((T, heads, vdim)), f64(start).copy(), 0
    values = f64(v).reshape(T, heads, v_cols)
    if ones:
        values = np.concatenate([values, np.ones((T, heads, 1)), np.zeros((T, heads, vdim - v_cols - 1))], axis=2)
    of_head = lambda t: np.repeat(f64(t).reshape(T, groups, dim), heads // groups, axis=1)
    for n, slot in zip(lengths, slots):
        part = slice(at, at + n)
        want[part] = scan_oracle(form, of_head(q)[part] * 0.5, of_head(k)[part], values[part], decay[part], factor[part], None, want_state[slot])
        at += n
    want += f64(skip)[:, None] * values
    ctx = SimpleNamespace(q_start=torch.tensor(np.cumsum([0] + lengths), dtype=torch.int32, device=DEV), max_q_len=max(lengths))
    state = SimpleNamespace(buffer=start.to(DEV), slots=torch.tensor(slots, dtype=torch.int32, device=DEV))
    out = torch.full((T, heads * vdim), float("nan"), device=DEV)
    kernels.gated_scan(q.to(DEV), k.to(DEV), v.to(DEV), None if z is None else z.to(DEV), None if bias is None else bias.to(DEV), ctx, state, out, heads,
                       groups, dim, vdim, status, q_scale=0.5, ones_col=ones, skip=skip.to(DEV), **more)
    assert int(status.item()) == 0
    # float32 recurrences of up to 145 steps and sums over up to 128 products of terms of both signs: some 300 roundings of 2^-24
    for got, expected in ((out.double().cpu().numpy().reshape(want.shape), want), (state.buffer.double().cpu().numpy(), want_state)):
        assert np.abs(got - expected).max() <= 2e-5 * max(1.0, np.abs(expected).max())


@pytest.mark.parametrize("chunk", [48, 192])
@pytest.mark.parametrize("form,dim,vdim,ones", [("channel", 128, 136, False), ("head", 64, 72, False), ("given", 128, 130, True)])
def test_gated_scan_16_tokens_at_a_time_in_chunks(status, monkeypatch, chunk, form, dim, vdim, ones):
    """The same in chunks of several steps of 16 tokens, portions that end within one, and in one chunk a portion (the rule takes one step a chunk there)."""
    from sprout_lm_b200 import kernels
    monkeypatch.setattr(kernels, "scan_mma_chunk", lambda *a, **k: chunk)
    test_gated_scan_16_tokens_at_a_time(status, form, 1.0, dim, vdim, ones)


@pytest.mark.parametrize("what,value", [("q", math.inf), ("k", math.inf), ("k", math.nan), ("v", -math.inf), ("v", math.nan), ("decay", math.nan),
                                        ("state", math.inf), ("state", math.nan)])
@pytest.mark.parametrize("form,dim,vdim", [("channel", 64, 72), ("channel", 128, 136), ("head", 128, 64), ("given", 64, 40)])
def test_gated_scan_values_that_are_not_finite(status, monkeypatch, form, dim, vdim, what, value):
    """An infinity or a NaN at the start, in the middle and at the end of 16 tokens, of a chunk and of a portion, through the walk on tensor cores: infinities and
    NaN come where the recurrence in turn (float64) has them; outputs before its 16 tokens, other columns (of a value or a state) and other requests keep their
    bits, outputs before it among its 16 tokens their value."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    monkeypatch.setattr(kernels, "scan_mma_chunk", lambda *a, **k: 48)
    heads, lengths, slots = 2, [17, 145, 66], [2, 0, 3]
    g = torch.Generator().manual_seed(dim + vdim)
    T, begin = sum(lengths), lengths[0]
    make = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
    clean = dict(q=make(T, dim), k=make(T, dim), v=make(T, heads * vdim), state=torch.randn(4, heads, dim, vdim, generator=g))
    # weak decays: over a chunk their product stays a float32, so that an infinite state stays one
    clean["decay"] = torch.rand(T, heads, generator=g) ** 0.1 if form == "given" else torch.randn(T, heads * (dim if form == "channel" else 1), generator=g)
    bias, factor, skip = torch.linspace(-1.0, 1.0, clean["decay"].shape[1]), torch.rand(T, heads, generator=g) + 0.5, torch.tensor([-0.5, 1.0])
    f64 = lambda t: t.double().numpy()

    def run(x):
        x = {name: t.to(DEV) for name, t in x.items()}
        more = dict(given=(x["decay"], factor.to(DEV))) if form == "given" else dict(per_head=True, a_log=torch.full((heads,), math.log(0.1), device=DEV)) if form == "head" \
            else dict(tau=10.0)
        ctx = SimpleNamespace(q_start=torch.tensor(np.cumsum([0] + lengths), dtype=torch.int32, device=DEV), max_q_len=max(lengths))
        state = SimpleNamespace(buffer=x["state"], slots=torch.tensor(slots, dtype=torch.int32, device=DEV))
        out = torch.full((T, heads * vdim), 7.0, device=DEV)
        z = (None, None) if form == "given" else (x["decay"], bias.to(DEV))
        kernels.gated_scan(x["q"], x["k"], x["v"], *z, ctx, state, out, heads, 1, dim, vdim, status, q_scale=0.5, skip=skip.to(DEV), **more)
        assert int(status.item()) == 0
        return out.cpu().view(T, heads, vdim), state.buffer.cpu()

    before, state_before = run(clean)
    for at in (0, 15, 24, 47, 48, 100, 144):
        x = {name: t.clone() for name, t in clean.items()}
        t = begin + at
        column = at % vdim
        if what == "state":
            x["state"][slots[1], 1, dim // 2, column] = value
            t = begin
        elif what == "v":
            x["v"][t, vdim + column] = value
        else:
            x[what][t, -1] = value
        got, state = run(x)
        with np.errstate(all="ignore"):
            z = f64(x["decay"]) + (0.0 if form == "given" else f64(bias))
            if form == "given":
                decay, weight = np.repeat(z[:, :, None], dim, axis=2), f64(factor)
            elif form == "head":
                weight = np.logaddexp(0.0, z)
                decay = np.repeat(np.exp(-0.1 * weight)[:, :, None], dim, axis=2)
            else:
                decay, weight = (1.0 / (1.0 + np.exp(-z.reshape(T, heads, dim)))) ** 0.1, np.ones((T, heads))
            want, want_state = np.zeros((T, heads, vdim)), f64(x["state"]).copy()
            of_heads = lambda name, part: np.repeat(f64(x[name][part])[:, None], heads, axis=1)
            first = 0
            for n, slot in zip(lengths, slots):
                part = slice(first, first + n)
                want[part] = scan_oracle(form, of_heads("q", part) * 0.5, of_heads("k", part), f64(x["v"][part]).reshape(n, heads, vdim), decay[part], weight[part], None,
                                         want_state[slot])
                first += n
            want += f64(skip)[:, None] * f64(x["v"]).reshape(T, heads, vdim)
        assert not np.isfinite(want).all()
        for result, expected in ((f64(got), want), (f64(state), want_state)):
            finite = np.isfinite(expected)
            assert (np.isnan(result) == np.isnan(expected)).all() and (result[np.isinf(expected)] == expected[np.isinf(expected)]).all()
            # as the walk over finite values, see above
            assert np.abs(result[finite] - expected[finite]).max() <= 2e-5 * max(1.0, np.abs(expected[finite]).max())
        for part in (slice(0, begin + (t - begin) // 16 * 16), slice(begin + lengths[1], T)):
            assert torch.equal(got[part], before[part])
        if what in ("v", "state"):
            keep = torch.ones(heads, vdim, dtype=torch.bool)
            keep[1, column] = False
            assert torch.equal(got[:, keep], before[:, keep]) and torch.equal(state.transpose(1, 2)[:, :, keep], state_before.transpose(1, 2)[:, :, keep])


@pytest.mark.parametrize("form", ["channel", "head", "floor", "bonus"])
@pytest.mark.parametrize("dim,vdim", [(16, 24), (64, 40), (128, 64), (256, 20), (40, 12)])
def test_float32_scan_keeps_its_bits_beside_a_long_portion(status, form, dim, vdim):
    """The 32-bit path adds in one order: a short request (walked whole alone, as a chunk beside a portion of 300 tokens) has the same bits both ways."""
    from types import SimpleNamespace
    from sprout_lm_b200 import kernels
    heads, lengths = 2, [33, 300, 1, 64]
    g = torch.Generator().manual_seed(dim)
    T = sum(lengths)
    starts = np.cumsum([0] + lengths)
    make = lambda *shape: torch.randn(*shape, generator=g).to(DEV)
    q, k, v, z = make(T, heads * dim), make(T, heads * dim), make(T, heads * vdim), make(T, heads if form == "head" else heads * dim)
    bias, first = make(heads if form == "head" else heads * dim), make(len(lengths), heads, dim, vdim)
    more = {"channel": dict(tau=2.0), "head": dict(per_head=True, a_log=make(heads)), "floor": dict(floor=torch.rand(heads * dim, generator=g).to(DEV)),
            "bonus": dict(bonus=make(heads * dim))}[form]

    def scan(requests):
        rows = torch.cat([torch.arange(starts[r], starts[r + 1]) for r in requests]).to(DEV)
        ctx = SimpleNamespace(q_start=torch.tensor(np.cumsum([0] + [lengths[r] for r in requests]), dtype=torch.int32, device=DEV),
                              max_q_len=max(lengths[r] for r in requests))
        state = SimpleNamespace(buffer=first.clone(), slots=torch.tensor(requests, dtype=torch.int32, device=DEV))
        out = torch.empty(len(rows), heads * vdim, device=DEV)
        kernels.gated_scan(q[rows], None if form == "floor" else k[rows], v[rows], z[rows], bias, ctx, state, out, heads, heads, dim, vdim, status, **more)
        return out, state.buffer
    together, states = scan([0, 1, 2, 3])
    for r in (0, 2, 3):
        alone, state = scan([r])
        assert torch.equal(alone, together[starts[r]:starts[r + 1]]) and torch.equal(state[r], states[r]), r
    assert int(status.item()) == 0


@pytest.mark.parametrize("heads,kv_heads,held,new", [(28, 4, [0, 0, 70], [64, 130, 61]), (8, 1, [0], [192]), (16, 16, [5, 0], [128, 177])])
def test_prompt_attention_of_head_size_128_both_kernels(status, heads, kv_heads, held, new):
    """Short contexts: the kernel that adds O up in registers (the step's longest context given) and the one in tensor memory (not given) against
    the float32-arithmetic kernel."""
    from sprout_lm_b200 import kernels
    case = build_paged_case(torch.bfloat16, heads, kv_heads, 128, 16, [h + n for h, n in zip(held, new)], new)
    outs = []
    for context in (max(h + n for h, n in zip(held, new)), 0):
        out = torch.full((case["T"], heads * 128), float("nan"), dtype=torch.bfloat16, device=DEV)
        kernels.attention_prefill(case["q"], case["k_cache"], case["v_cache"], case["table"], case["q_start"], case["positions"], out, heads, kv_heads, 128,
                                  status, variant="tcgen05", max_context=context)
        outs.append(out.float())
    want = torch.empty(case["T"], heads * 128, dtype=torch.bfloat16, device=DEV)
    kernels.attention_simple(case["q"], case["k_cache"], case["v_cache"], case["table"], case["seq_of_token"], case["positions"], want, heads, kv_heads, 128, status)
    for out in outs:
        # probabilities and the result rounded to 8 bits
        assert (out - want.float()).norm() <= 6e-3 * want.float().norm()
    assert int(status.item()) == 0
