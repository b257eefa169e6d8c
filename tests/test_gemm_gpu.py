"""The whole-prompt path on the GPU: the tensor-core projection GEMM (attn_gemm_f16) and the row-wise steps around it,
against the engine's CPU functions (matmul(), rmsnorm(), rope() of include/kernels_cpu.hpp and the SwiGLU of
src/model/block.cpp:206-210) applied one token at a time, the way the engine processes a prompt
(tools/infer.cpp:271-274)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def A(built_lib, pkg):
    import torch
    assert torch.cuda.is_available()
    from llm_infer_b200 import attention
    return attention


def _pair(x):
    """fp32 array -> (hi, lo) fp16 arrays the way the device writes them."""
    x = np.clip(x, -65504, 65504).astype(np.float32)
    hi = x.astype(np.float16)
    lo = (x - hi.astype(np.float32)).astype(np.float16)
    return hi, lo


@pytest.mark.parametrize("m,n_out,k", [(1, 32, 64), (127, 96, 128), (128, 256, 64), (129, 288, 192), (300, 544, 1024),
                                       (1000, 4096, 4096), (513, 6144, 256)])
def test_gemm_against_float64_and_accumulate(A, m, n_out, k):
    import torch
    rng = np.random.default_rng(m + n_out + k)
    x = rng.standard_normal((m, k), dtype=np.float32)
    w = (rng.standard_normal((n_out, k), dtype=np.float32) * k ** -0.5).astype(np.float16)
    hi, lo = _pair(x)
    a64 = hi.astype(np.float64) + lo.astype(np.float64)
    want = a64 @ w.astype(np.float64).T
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hid, lod, wd = (torch.from_numpy(t).cuda() for t in (hi, lo, w))
    out = torch.full((m, n_out), float("nan"), device="cuda")
    A.gemm_f16(hid, lod, wd, out=out, status=status)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    scale = np.abs(want).max()
    assert np.isfinite(got).all()
    # fp32 accumulation inside the tensor cores over k / 16 steps: a few 1e-6 of the largest output per 64 columns of k
    tol = 4e-6 * scale * (k / 64) ** 0.5
    assert np.abs(got - want).max() <= tol, "value + residual product"
    # accumulate on top, without the residual term, into a strided output
    wide = torch.zeros((m, n_out + 32), device="cuda")
    view = wide[:, :n_out]
    view.copy_(out)
    A.gemm_f16(hid, None, wd, out=view, accumulate=True, status=status)
    torch.cuda.synchronize()
    want2 = want + hi.astype(np.float64) @ w.astype(np.float64).T
    assert np.abs(view.cpu().numpy() - want2).max() <= 2 * tol
    assert bool((wide[:, n_out:] == 0).all()), "nothing written past the row"
    assert int(status.item()) == 0


def _truncation_bound(k, products, scale):
    """The tensor cores drop what lies below the accumulator's last bit once per k-step of 16 and product: at most
    2^-23 of the running sum each, which stays below the largest output here."""
    return (k / 16 * products * 2.0 ** -23 + 2.0 ** -20) * scale


# one token, around 128 and 256 (single CTA / pair), several bands of rows, widths that leave part of a tile
@pytest.mark.parametrize("m,n_out,k", [(1, 32, 64), (128, 96, 128), (129, 160, 192), (256, 256, 64), (257, 4128, 256),
                                       (700, 1056, 512), (2500, 416, 14336)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_gemm_with_paired_weights(A, m, n_out, k, swiglu):
    """attn_gemm_pair against float64: three products in one pass, accumulate, and the SwiGLU epilogue."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n_out + k)
    x = torch.randn((m, k), generator=g, device="cuda")
    w = torch.randn((n_out * (2 if swiglu else 1), k), generator=g, device="cuda") * k ** -0.5
    split = lambda t: (t.half(), (t - t.half().float()).half())  # noqa: E731
    (ah, al), (wh, wl) = split(x), split(w)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    a64, w64 = ah.double() + al.double(), wh.double() + wl.double()
    prod = a64 @ w64.T  # the product of the two residuals, 2^-24 of a term, is not part of the result
    tol = _truncation_bound(k, 1, float(prod.abs().max()))
    if swiglu:
        out = tuple(torch.full((m, n_out), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
        A.gemm_pair((ah, al), (wh, wl), out=out, swiglu=True, status=status)
        gate, up = prod[:, :n_out], prod[:, n_out:]
        want = gate / (1 + torch.exp(-gate)) * up
        # d(silu(g) u) <= 1.1 |u| dg + |g| du, and the pair's own 2^-21 of the value
        bound = 1.1 * tol * (up.abs() + gate.abs()) + 2.0 ** -20 * want.abs() + 2.0 ** -24
        assert bool(((out[0].double() + out[1].double() - want).abs() <= bound).all())
        only = tuple(torch.empty_like(t) for t in out)
        A.gemm_pair((ah, None), (wh, None), out=only, swiglu=True, status=status)
        p1 = ah.double() @ wh.double().T
        gate, up = p1[:, :n_out], p1[:, n_out:]
        want = gate / (1 + torch.exp(-gate)) * up
        bound = 1.1 * tol * (up.abs() + gate.abs()) + 2.0 ** -20 * want.abs() + 2.0 ** -24
        assert bool(((only[0].double() + only[1].double() - want).abs() <= bound).all())
    else:
        wide = torch.zeros((m, n_out + 32), device="cuda")
        A.gemm_pair((ah, al), (wh, wl), out=wide[:, :n_out], status=status)
        assert float((wide[:, :n_out].double() - prod).abs().max()) <= tol
        assert bool((wide[:, n_out:] == 0).all()), "nothing written past the row"
        A.gemm_pair((ah, None), (wh, wl), out=wide[:, :n_out], accumulate=True, status=status)
        want = prod + ah.double() @ w64.T
        assert float((wide[:, :n_out].double() - want).abs().max()) <= 3 * tol
    assert int(status.item()) == 0


# Several tiles per CTA (the tests above give each at most one): accumulators handed back and forth between the MMAs and the
# epilogue, and ring and barrier phases that run on over the tiles. Tiles in all / at once, at 148 SMs: pairs of CTAs 224 and
# 256 wide with rows and columns that end inside a tile, 4 to 7 times (one accumulator at a time with three products, else
# two); single CTAs 224 wide, 2 to 4 times; single CTAs (three products) or pairs 256 wide, 8 to 17 times over several bands;
# 128 and 96 wide, 3 times, two accumulators with three products.
@pytest.mark.parametrize("m,n_out,k", [(2500, 6144, 128), (2500, 6176, 128), (100, 57408, 128), (2600, 14336, 64),
                                       (40001, 128, 64), (40001, 96, 128)])
@pytest.mark.parametrize("form", ["f16", "pair", "swiglu", "swiglu pair"])
def test_gemm_several_tiles_per_cta(A, m, n_out, k, form):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n_out + k)
    swiglu, paired = "swiglu" in form, "pair" in form
    x = torch.randn((m, k), generator=g, device="cuda")
    w = torch.randn((n_out * (2 if swiglu else 1), k), generator=g, device="cuda") * k ** -0.5
    split = lambda t: (t.half(), (t - t.half().float()).half())  # noqa: E731
    (ah, al), (wh, wl) = split(x), split(w)
    w_pair = (wh, wl if paired else None)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = tuple(torch.empty((m, n_out), dtype=torch.float16, device="cuda") for _ in range(2)) if swiglu else \
        torch.ones((m, n_out), device="cuda")
    if swiglu:
        A.gemm_pair((ah, al), w_pair, out=out, swiglu=True, status=status)
    elif paired:
        A.gemm_pair((ah, al), w_pair, out=out, accumulate=True, status=status)
    else:
        A.gemm_f16(ah, al, wh, out=out, accumulate=True, status=status)
    w64 = wh.double() + wl.double() if paired else wh.double()
    for r in range(0, m, 4000):  # (float64 blocks of rows)
        prod = (ah[r:r + 4000].double() + al[r:r + 4000].double()) @ w64.T
        tol = _truncation_bound(k, 1 if paired else 2, float(prod.abs().max()))
        if swiglu:
            gate, up = prod[:, :n_out], prod[:, n_out:]
            want = gate / (1 + torch.exp(-gate)) * up
            bound = 1.1 * tol * (up.abs() + gate.abs()) + 2.0 ** -20 * want.abs() + 2.0 ** -24
            assert bool(((out[0][r:r + 4000].double() + out[1][r:r + 4000].double() - want).abs() <= bound).all())
        else:  # the sum with what was there rounds once more
            assert float((out[r:r + 4000].double() - 1.0 - prod).abs().max()) <= tol + 2.0 ** -24 * (float(prod.abs().max()) + 1)
    assert int(status.item()) == 0


def _q8_blocks(g, rows, k):
    import torch
    q = torch.randint(-127, 128, (rows, k // 32, 32), generator=g, device="cuda", dtype=torch.int8)
    d = (torch.rand((rows, k // 32, 1), generator=g, device="cuda") * k ** -0.5 / 64).half()
    blocks = torch.empty((rows, k // 32, 34), dtype=torch.uint8, device="cuda")
    blocks[..., :2], blocks[..., 2:] = d.view(torch.uint8), q.view(torch.uint8)
    return blocks.view(rows, -1), (d.double() * q.double()).view(rows, k)


# Rows and tokens around the tiles (64 and 128 tokens, 128 to 512 rows), k of two blocks, an odd number of block pairs and
# no multiple of eight blocks, several tiles per CTA over several bands; all forms: one or two row parts, single CTAs and pairs.
@pytest.mark.parametrize("m,n_out,k", [(1, 1, 64), (63, 130, 192), (128, 512, 256), (129, 513, 320), (700, 1056, 512),
                                       (2500, 6200, 64), (9000, 520, 128), (500, 416, 14336), (40, 20000, 64)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_gemm_q8_0_against_float64(A, m, n_out, k, swiglu):
    """attn_expand_q8_0 exactly, and attn_gemm_q8_0 against float64: a block's sum is cut once per MMA of 16 (four of them,
    2^-23 of it at most), and the scaled sums of k / 32 blocks are rounded once each in fp32."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n_out + k)
    w, w64 = _q8_blocks(g, n_out * (2 if swiglu else 1), k)
    q, d = A.expand_q8_0(w)
    assert torch.equal((q.view(-1, k // 32, 32).double() * d[:, :k // 32, None].double()).view(-1, k), w64)
    x = torch.randn((m, k), generator=g, device="cuda")
    a = (x.half(), (x - x.half().float()).half())
    a64 = a[0].double() + a[1].double()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    prod = a64 @ w64.T
    # k / 32 additions, each off by 2^-24 of the running sum at most, and 4 * 2^-23 of the blocks' sums; a running sum of terms
    # of random sign stays within four of its standard deviations, |a| |w| / sqrt(k), or the largest result
    sums = max(float(prod.abs().max()), 4 * float(a64.norm(dim=1).max() * w64.norm(dim=1).max()) * k ** -0.5)
    tol = (k / 32 * 2.0 ** -24 + 2.0 ** -20) * sums
    if swiglu:
        out = tuple(torch.full((m, n_out), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
        A.gemm_q8_0(a, (q, d), out=out, swiglu=True, status=status)
        gate, up = prod[:, :n_out], prod[:, n_out:]
        want = gate / (1 + torch.exp(-gate)) * up
        bound = 1.1 * tol * (up.abs() + gate.abs()) + 2.0 ** -20 * want.abs() + 2.0 ** -24
        assert bool(((out[0].double() + out[1].double() - want).abs() <= bound).all())
    else:
        wide = torch.zeros((m, n_out + 3), device="cuda")
        A.gemm_q8_0(a, (q, d), out=wide[:, :n_out], status=status)
        assert float((wide[:, :n_out].double() - prod).abs().max()) <= tol
        assert bool((wide[:, n_out:] == 0).all()), "nothing written past the row"
        A.gemm_q8_0(a, (q, d), out=wide[:, :n_out], accumulate=True, status=status)
        assert float((wide[:, :n_out].double() - 2 * prod).abs().max()) <= 3 * tol
    assert int(status.item()) == 0


@pytest.mark.parametrize("m,n_out,k,swiglu", [(1003, 4096, 4096, False), (700, 2048, 14336, True)])
def test_gemm_q8_0_hands_its_accumulators_back_in_order(A, m, n_out, k, swiglu):
    """Four accumulators go round between the MMAs and the warps that read them, once per block of 32: every element is one fixed
    order of sums, so a hundred calls agree bit for bit, and so does a call of which only a token tile's rows are asked for."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(k)
    w, _ = _q8_blocks(g, n_out * (2 if swiglu else 1), k)
    planes = A.expand_q8_0(w)
    x = torch.randn((m, k), generator=g, device="cuda")
    pair = (x.half(), (x - x.half().float()).half())

    def call(rows):
        shape = (rows, n_out)
        out = tuple(torch.empty(shape, dtype=torch.float16, device="cuda") for _ in range(2)) if swiglu else torch.empty(shape, device="cuda")
        A.gemm_q8_0(tuple(t[:rows] for t in pair), planes, out=out, swiglu=swiglu)
        return torch.cat([t.float() for t in out]) if swiglu else out, out

    first, parts = call(m)
    for _ in range(100):
        assert torch.equal(call(m)[0], first)
    few = call(64)[1]  # other tiles, single CTAs or pairs as the cost rule has it
    for got, want in zip(few, parts) if swiglu else [(few, parts)]:
        assert torch.equal(got, want[:64])


def test_gemm_rows_equal_the_engine_matmul(A, checker):
    """Each token's row of the GEMM against the engine's own per-token matmul() on the fp32 activations."""
    import torch
    rng = np.random.default_rng(7)
    m, n_out, k = 37, 512, 1024
    x = rng.standard_normal((m, k), dtype=np.float32)
    w = (rng.standard_normal((n_out, k), dtype=np.float32) * 0.03).astype(np.float16)
    hi, lo = A.split_pair(torch.from_numpy(x).cuda())
    out = torch.empty((m, n_out), device="cuda")
    A.gemm_f16(hi, lo, torch.from_numpy(w).cuda(), out=out)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for t in (0, 5, 36):
        want = checker.matmul_clip(x[t], w, 0.0)  # itself a sequential fp32 sum over 1024 terms (~1e-5 of its own)
        np.testing.assert_allclose(got[t], want, rtol=0, atol=3e-5 * np.abs(want).max())


def test_row_steps_against_the_cpu_functions(A, checker, port, pkg):
    import torch
    from llm_infer_b200 import quant
    rng = np.random.default_rng(9)
    rows, dim, hidden = 21, 1024, 1536
    x = rng.standard_normal((rows, dim), dtype=np.float32) * 2
    wt = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    hi, lo = A.rmsnorm_pair(torch.from_numpy(x).cuda(), torch.from_numpy(wt).cuda(), 1e-5)
    got = hi.float().cpu().numpy().astype(np.float64) + lo.float().cpu().numpy()
    for r in (0, 20):
        want = checker.rmsnorm(x[r], wt, 1e-5)
        assert np.abs(got[r] - want).max() <= 4e-6 * np.abs(want).max()
    gu = rng.standard_normal((rows, 2 * hidden), dtype=np.float32) * 3
    hi, lo = A.swiglu_pair(torch.from_numpy(gu).cuda())
    got = hi.float().cpu().numpy().astype(np.float64) + lo.float().cpu().numpy()
    want = port.swiglu(gu[:, :hidden].copy(), gu[:, hidden:].copy())
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
    wq = quant.quantize_q8_0(rng.standard_normal((48, 256), dtype=np.float32) * 0.05)
    hi, lo = A.dequant_q8_0_pair(torch.from_numpy(wq).cuda())
    got = hi.float().cpu().numpy().astype(np.float64) + lo.float().cpu().numpy()
    want = quant.dequantize_q8_0(wq)
    assert np.abs(got - want).max() <= 2.0 ** -21 * np.abs(want).max()
    idx = torch.tensor([20, 0, 7], dtype=torch.int32, device="cuda")
    out = torch.empty((3, dim), device="cuda")
    A.gather_rows(torch.from_numpy(x).cuda(), idx, out=out)
    assert np.array_equal(out.cpu().numpy(), x[[20, 0, 7]])


@pytest.mark.parametrize("D,rot,clip", [(128, 128, 0.0), (128, 64, 1.5), (64, 64, 0.0)])
def test_rope_prompt_fills_the_caches_like_the_per_token_loop(A, checker, D, rot, clip):
    """Two sequences of 5 and 3 prompt tokens packed into 8 rows: rotated q, and the K / V cache rows, against the
    engine's rope + insert (src/model/block.cpp:140-148) run token by token."""
    import torch
    rng = np.random.default_rng(D + rot)
    H, Hkv, T, theta = 4, 2, 16, 500000.0
    lens = [5, 3]
    tokens = sum(lens)
    qkv = rng.standard_normal((tokens, (H + 2 * Hkv) * D), dtype=np.float32) * 2
    seq = np.repeat(np.arange(2, dtype=np.int32), lens)
    pos = np.concatenate([np.arange(n, dtype=np.int32) for n in lens])
    kc = torch.zeros((2, T, Hkv, D), dtype=torch.float16, device="cuda")
    vc = torch.zeros_like(kc)
    q16 = torch.empty((tokens, H, D), dtype=torch.float16, device="cuda")
    A.rope_prompt(torch.from_numpy(qkv).cuda(), q16, kc, vc, torch.from_numpy(seq).cuda(), torch.from_numpy(pos).cuda(),
                  n_heads=H, theta=theta, rotary_dim=0 if rot == D else rot, qkv_clip=clip)
    torch.cuda.synchronize()
    src = np.clip(qkv, -clip, clip) if clip > 0 else qkv
    want_k = np.zeros((2, T, Hkv, D), dtype=np.float16)
    want_v = np.zeros_like(want_k)
    for t in range(tokens):
        q = src[t, :H * D].reshape(H, D)
        k = src[t, H * D:(H + Hkv) * D].reshape(Hkv, D)
        v = src[t, (H + Hkv) * D:].reshape(Hkv, D)
        q_rot, _ = checker.rope_kv_insert(q, k, v, want_k[seq[t]], want_v[seq[t]], int(pos[t]), int(pos[t]), theta=theta,
                                          rotary_dim=rot)
        got_q = q16[t].float().cpu().numpy()
        assert np.abs(got_q - q_rot).max() <= 2.0 ** -10 * max(1.0, np.abs(q_rot).max())
    gk, gv = kc.cpu().numpy(), vc.cpu().numpy()
    assert np.array_equal(gv.view(np.uint16), want_v.view(np.uint16))
    diff = np.abs(gk.astype(np.float32) - want_k.astype(np.float32))
    assert (diff <= np.maximum(np.abs(want_k.astype(np.float32)), 2.0 ** -14) * 2.0 ** -10).all()
    assert (gk.view(np.uint16) == want_k.view(np.uint16)).mean() > 0.97
