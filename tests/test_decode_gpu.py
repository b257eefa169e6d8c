"""GPU parity of the split-KV decode path, called through the C ABI, against the
CPU checker (the engine's attn(), include/kernels_cpu.hpp:140-167) on identical
seeded inputs. Tolerance: max abs 2e-3, max rel 1e-2 (relative error measured
against max(|ref|, 1% of the RMS of ref))."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def attention(built_lib, pkg):
    import torch
    assert torch.cuda.is_available()
    from llm_infer_b200 import attention as a
    return a


@pytest.fixture(scope="module")
def wl(pkg):
    return pkg.workloads


def _rand(wl, seed, B, H, Hkv, D, T, q_dtype="f32", kv_dtype="f16"):
    shape = wl.DecodeShape("t", seed, B, H, Hkv, D, T, q_dtype, kv_dtype)
    return wl.decode_inputs(shape)


def _oracle(wl, checker, q, k, v, q_dtype, kv_dtype, kv_len=None):
    return checker.attn_decode(wl.widen(q, q_dtype), wl.as_f16_for_oracle(k, kv_dtype),
                               wl.as_f16_for_oracle(v, kv_dtype),
                               None if kv_len is None else np.asarray(kv_len, np.uint32))


def test_golden_vectors(attention, wl):
    from gpu_util import check_close, run_decode
    g = np.load(os.path.join(GOLDEN, "decode_golden.npz"))
    for name in sorted({k.split(".")[0] for k in g.files}):
        lens = g[f"{name}.kv_len"]
        got = run_decode(attention, g[f"{name}.q"], g[f"{name}.k"], g[f"{name}.v"], kv_len=lens)
        check_close(wl, got, g[f"{name}.o"], name)


def test_c1_tinyllama_shape(attention, wl, checker):
    from gpu_util import check_close, run_decode
    q, k, v = wl.decode_inputs(wl.C1)
    got = run_decode(attention, q, k, v)
    check_close(wl, got, checker.attn_decode(q, k, v), "C1")


def test_c2_llama3_batched_full_size(attention, wl, checker):
    from gpu_util import check_close, run_decode
    q, k, v = wl.decode_inputs(wl.C2)
    got = run_decode(attention, q, k, v, q_dtype="f16")
    want = checker.attn_decode(q.astype(np.float32), k, v)
    max_abs, max_rel = check_close(wl, got, want, "C2")
    print(f"C2 max_abs={max_abs:.3e} max_rel={max_rel:.3e}")


def test_c4_long_context_single_gpu(attention, wl, checker):
    from gpu_util import check_close, run_decode
    q, k, v = wl.decode_inputs(wl.C4)
    got, lse = run_decode(attention, q, k, v, q_dtype="f16", lse=True)
    want = checker.attn_decode(q.astype(np.float32), k, v)
    max_abs, max_rel = check_close(wl, got, want, "C4")
    print(f"C4 max_abs={max_abs:.3e} max_rel={max_rel:.3e}")
    assert np.isfinite(lse).all()


@pytest.mark.parametrize("kv_len", [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 1000, 4095, 4097])
def test_edge_lengths(attention, wl, checker, kv_len):
    from gpu_util import check_close, run_decode
    q, k, v = _rand(wl, 100 + kv_len, 2, 32, 8, 128, kv_len)
    got = run_decode(attention, q, k, v)
    check_close(wl, got, _oracle(wl, checker, q, k, v, "f32", "f16"), f"kv_len={kv_len}")


@pytest.mark.parametrize("H,Hkv,D", [(4, 4, 64), (8, 1, 128), (8, 2, 64), (16, 4, 128), (32, 4, 64), (64, 8, 128),
                                     (32, 2, 128), (16, 16, 64), (48, 24, 128), (12, 6, 64), (5, 5, 128)])
def test_head_configurations(attention, wl, checker, H, Hkv, D):
    from gpu_util import check_close, run_decode
    q, k, v = _rand(wl, H * 1000 + Hkv * 10 + D, 3, H, Hkv, D, 333)
    got = run_decode(attention, q, k, v)
    check_close(wl, got, _oracle(wl, checker, q, k, v, "f32", "f16"), f"H={H} Hkv={Hkv} D={D}")


def test_ragged_batch_including_empty_sequence(attention, wl, checker):
    from gpu_util import check_close, run_decode
    lens = [1, 700, 0, 64, 699, 5, 333, 128]
    q, k, v = _rand(wl, 7, len(lens), 32, 8, 128, 700)
    got, lse = run_decode(attention, q, k, v, kv_len=lens, lse=True)
    want = _oracle(wl, checker, q, k, v, "f32", "f16", lens)
    check_close(wl, got, want, "ragged")
    assert np.array_equal(got[2], np.zeros_like(got[2]))  # empty sequence -> zeros, as the CPU loop gives
    assert np.isneginf(lse[2]).all() and np.isfinite(np.delete(lse, 2, axis=0)).all()


@pytest.mark.parametrize("q_dtype,kv_dtype,out_dtype", [("f16", "f16", "f32"), ("bf16", "f16", "f32"),
                                                         ("f32", "bf16", "f32"), ("bf16", "bf16", "bf16"),
                                                         ("f16", "f16", "f16")])
def test_dtypes(attention, wl, checker, q_dtype, kv_dtype, out_dtype):
    from gpu_util import run_decode
    q, k, v = _rand(wl, 11, 2, 32, 8, 128, 777, q_dtype, kv_dtype)
    got = run_decode(attention, q, k, v, q_dtype=q_dtype, kv_dtype=kv_dtype, out_dtype=out_dtype)
    want = _oracle(wl, checker, q, k, v, q_dtype, kv_dtype)
    max_abs, max_rel = wl.error_metrics(got, want)
    # 16-bit outputs carry their own rounding (bf16: 2^-9 relative)
    rel_tol = {"f32": wl.REL_TOL, "f16": wl.REL_TOL, "bf16": 1.5e-2}[out_dtype]
    assert max_abs <= wl.ABS_TOL and max_rel <= rel_tol, (max_abs, max_rel)


def test_lse_output(attention, wl, port):
    from gpu_util import run_decode
    q, k, v = _rand(wl, 12, 1, 8, 2, 64, 200)
    _, lse = run_decode(attention, q, k, v, lse=True)
    for h in (0, 3, 7):
        m, z, _ = port.state_from_rows(q[0, h], k[0], v[0], h // 4, 0, 200)
        assert abs(lse[0, h] - (m + np.log(z))) < 1e-4


def test_strided_cache_with_spare_capacity(attention, wl, checker):
    """Cache rows wider than n_kv_heads*head_dim and longer than kv_len, as a preallocated cache has."""
    import torch
    from gpu_util import check_close, to_device
    B, H, Hkv, D, T, cap = 2, 32, 8, 128, 300, 512
    q, k, v = _rand(wl, 13, B, H, Hkv, D, T)
    kbig = torch.zeros((B, cap, Hkv + 1, D), dtype=torch.float16, device="cuda")
    vbig = torch.full((B, cap, Hkv + 1, D), float("nan"), dtype=torch.float16, device="cuda")
    kbig[:, :T, :Hkv] = to_device(k, "f16")
    vbig[:, :T, :Hkv] = to_device(v, "f16")
    out = attention.attn_decode(to_device(q, "f32"), kbig[:, :, :Hkv], vbig[:, :, :Hkv], T)
    torch.cuda.synchronize()
    check_close(wl, out.cpu().numpy(), checker.attn_decode(q, k, v), "strided")


def test_bitwise_deterministic_and_canaries(attention, wl):
    import torch
    from gpu_util import to_device
    q, k, v = _rand(wl, 14, 4, 32, 8, 128, 1500)
    qd, kd, vd = to_device(q, "f32"), to_device(k, "f16"), to_device(v, "f16")
    ws = attention.DecodeWorkspace(4, 32, 8, 128)
    padded = torch.full((4 * 32 * 128 + 512,), float("nan"), dtype=torch.float32, device="cuda")
    out = padded[256:256 + 4 * 32 * 128].view(4, 32, 128)
    attention.attn_decode(qd, kd, vd, out=out, workspace=ws)
    first = out.clone()
    for _ in range(3):
        attention.attn_decode(qd, kd, vd, out=out, workspace=ws)
        assert torch.equal(out, first)
    torch.cuda.synchronize()
    assert torch.isnan(padded[:256]).all() and torch.isnan(padded[-256:]).all()  # nothing written outside o
    assert int(ws.status.item()) == 0


def test_early_streaming_after_an_appending_kernel(attention, wl, checker):
    """kv_early: the split pass may start its K/V copies before the kernel in front of it (here the rotary kernel that
    appends the token's row) has finished, for every tile that cannot hold that row. Back-to-back steps through the
    programmatic-launch chain, ragged and uniform lengths, must give the result of the plain call and of the CPU."""
    import torch
    from gpu_util import check_close, to_device
    B, H, Hkv, D, T = 3, 32, 8, 128, 700
    q, k, v = _rand(wl, 77, B, H, Hkv, D, T, "f32", "f16")
    rng = np.random.default_rng(78)
    lens = np.array([700, 33, 257], dtype=np.int32)
    kd, vd = to_device(k, "f16"), to_device(v, "f16")
    knew = rng.standard_normal((B, Hkv, D), dtype=np.float32)
    vnew = rng.standard_normal((B, Hkv, D), dtype=np.float32)
    pos = torch.from_numpy(lens - 1).cuda()
    lens_d = torch.from_numpy(lens).cuda()
    ws = attention.DecodeWorkspace(B, H, Hkv, D)
    outs = []
    for early in (False, True, True):
        kc, vc = kd.clone(), vd.clone()
        q_rot = attention.rope_kv_insert(torch.from_numpy(q).cuda(), torch.from_numpy(knew).cuda(),
                                         torch.from_numpy(vnew).cuda(), kc, vc, pos, pos, theta=10000.0)
        outs.append(attention.attn_decode(q_rot, kc, vc, lens_d, workspace=ws, kv_early=early))
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2])
    want = checker.attn_decode(q_rot.cpu().numpy(), kc.cpu().numpy(), vc.cpu().numpy(), lens.astype(np.uint32))
    check_close(wl, outs[1].cpu().numpy(), want, "kv_early after rope insert")
    assert int(ws.status.item()) == 0


def test_length_beyond_the_cache_is_clamped_and_reported(attention, wl, checker):
    """A corrupted kv_len[] entry larger than the cache: the kernels clamp it to the stated capacity and raise
    ATTN_STATUS_BAD_SHAPE instead of reading past the cache."""
    import torch
    from gpu_util import check_close, to_device
    q, k, v = _rand(wl, 91, 2, 32, 8, 128, 300)
    lens = torch.tensor([100, 5000], dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(2, 32, 8, 128)
    out = attention.attn_decode(to_device(q, "f32"), to_device(k, "f16"), to_device(v, "f16"), lens, workspace=ws)
    torch.cuda.synchronize()
    assert int(ws.status.item()) == 2  # ATTN_STATUS_BAD_SHAPE
    want = checker.attn_decode(q, k, v, np.array([100, 300], np.uint32))
    check_close(wl, out.cpu().numpy(), want, "clamped length")


# The split pass and its merge serve every generation step, long contexts and sharded calls; short calls like those of the two
# tests above take the clusters, so the two-launch form is asked for here in both ways there are. Prepared words are what a Q8_0
# generation step has the attention write.
@pytest.mark.parametrize("words", [False, True])
@pytest.mark.parametrize("form", ["two_pass", "max_ctas"])
@pytest.mark.parametrize("H,Hkv,D,lens", [(32, 8, 128, [700, 33, 257]), (18, 2, 64, [1, 700, 130])])
def test_two_launches_behind_an_appending_kernel(attention, wl, checker, H, Hkv, D, lens, form, words):
    import torch
    from gpu_util import check_close, to_device
    B, T = 3, 700
    q, k, v = _rand(wl, 177, B, H, Hkv, D, T, "f32", "f16")
    rng = np.random.default_rng(178)
    new = [torch.from_numpy(rng.standard_normal((B, Hkv, D), dtype=np.float32)).cuda() for _ in range(2)]
    qd, kd, vd = torch.from_numpy(q).cuda(), to_device(k, "f16"), to_device(v, "f16")
    lens_d = torch.tensor(lens, dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(B, H, Hkv, D)
    kw = {"two_pass": True} if form == "two_pass" else {"max_ctas": torch.cuda.get_device_properties(0).multi_processor_count}
    outs = []
    for early in (False, True, True):
        kc, vc = kd.clone(), vd.clone()
        q_rot = attention.rope_kv_insert(qd.clone(), *new, kc, vc, lens_d - 1, lens_d - 1, theta=10000.0)
        out = torch.empty((B, H, D), dtype=torch.int32 if words else torch.float32, device="cuda")
        before = attention.kernel_launch_count()
        attention.attn_decode(q_rot, kc, vc, lens_d, out=out, workspace=ws, kv_early=early, **kw)
        assert attention.kernel_launch_count() - before == 2
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2])
    got = outs[1]
    if words:  # {hi(x0,x1), hi(x2,x3), lo(x0,x1), lo(x2,x3)} of four elements
        h = got.view(torch.float16).view(B, H, D // 4, 2, 4).float()
        got = (h[..., 0, :] + h[..., 1, :]).reshape(B, H, D)
    want = checker.attn_decode(q_rot.cpu().numpy(), kc.cpu().numpy(), vc.cpu().numpy(), np.array(lens, np.uint32))
    check_close(wl, got.cpu().numpy(), want, "two launches behind rope insert")
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("kw", [{"two_pass": True}, {"max_ctas": 148}, {"two_pass": True, "kv_early": True}])
def test_two_launches_clamp_and_report_a_length_beyond_the_cache(attention, wl, checker, kw):
    import torch
    from gpu_util import check_close, to_device
    q, k, v = _rand(wl, 91, 2, 32, 8, 128, 300)
    lens = torch.tensor([100, 5000], dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(2, 32, 8, 128)
    before = attention.kernel_launch_count()
    out = attention.attn_decode(to_device(q, "f32"), to_device(k, "f16"), to_device(v, "f16"), lens, workspace=ws, **kw)
    assert attention.kernel_launch_count() - before == 2
    assert int(ws.status.item()) == 2  # ATTN_STATUS_BAD_SHAPE
    check_close(wl, out.cpu().numpy(), checker.attn_decode(q, k, v, np.array([100, 300], np.uint32)), "clamped length")


@pytest.mark.parametrize("two_pass", [False, True])
@pytest.mark.parametrize("H,Hkv,D", [(32, 8, 128), (14, 2, 64)])
def test_an_output_off_its_16_byte_boundary(attention, wl, H, Hkv, D, two_pass):
    """fp32 results that start 4 bytes behind a boundary: element stores in the merges, the same bits, nothing beside them."""
    import torch
    from gpu_util import to_device
    q, k, v = _rand(wl, H, 2, H, Hkv, D, 333)
    qd, kd, vd = to_device(q, "f32"), to_device(k, "f16"), to_device(v, "f16")
    ws = attention.DecodeWorkspace(2, H, Hkv, D)
    want = attention.attn_decode(qd, kd, vd, workspace=ws, two_pass=two_pass)
    flat = torch.full((2 * H * D + 5,), -7.0, device="cuda")
    out = flat[1:1 + 2 * H * D].view(2, H, D)
    before = attention.kernel_launch_count()
    attention.attn_decode(qd, kd, vd, out=out, workspace=ws, two_pass=two_pass)
    assert attention.kernel_launch_count() - before == 1 + two_pass
    assert torch.equal(out, want) and bool((flat[:1] == -7).all()) and bool((flat[1 + 2 * H * D:] == -7).all())
    assert int(ws.status.item()) == 0


def test_checking_build_runs_clean(pkg, wl, checker, tmp_path):
    """The -DATTN_BOUNDS_CHECK build (the decode passes verify their workspace indices and report ATTN_STATUS_BAD_INDEX
    instead of accessing) gives the same results with no status bit on uniform, ragged and single-long-sequence
    shapes, through attn_decode and through the engine's single-launch kernel symbol. Runs in a child process because the library is chosen when the binding is first loaded."""
    import subprocess
    import sys
    from conftest import ROOT
    lib = pkg.build.build_library(check=True)
    code = f"""
import sys, numpy as np, torch
sys.path.insert(0, {ROOT!r}); sys.path.insert(0, {ROOT!r} + '/tests')
from conftest import load_package
pkg = load_package()
from llm_infer_b200 import attention, binding
assert binding.LIB_PATH.endswith('_check.so')
import oracle
wl = pkg.workloads
for (B, T, lens) in ((3, 700, [700, 1, 333]), (1, 20000, None), (16, 512, None)):
    q, k, v = wl.decode_inputs(wl.DecodeShape('c', 5, B, 32, 8, 128, T, 'f32', 'f16'))
    ws = attention.DecodeWorkspace(B, 32, 8, 128)
    l = None if lens is None else torch.tensor(lens, dtype=torch.int32, device='cuda')
    out = attention.attn_decode(torch.from_numpy(q).cuda(), torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda(), l, workspace=ws)
    torch.cuda.synchronize()
    assert int(ws.status.item()) == 0, ws.status.item()
    want = oracle.best().attn_decode(q, k, v, None if lens is None else np.array(lens, np.uint32))
    a, r = wl.error_metrics(out.cpu().numpy(), want)
    assert a <= wl.ABS_TOL and r <= wl.REL_TOL, (a, r)
# the engine's kernel symbol (single launch; two-level merge on the long sequence)
import ctypes as C
lib = binding.load()
n = lib.attention_workspace_bytes(32, 8, 128)
wsb = torch.zeros(n, dtype=torch.uint8, device='cuda')
stream = torch.cuda.current_stream().cuda_stream
assert lib.attention_configure(32, 8, 128, 0.0, wsb.data_ptr(), n, stream) == 0
for T in (300, 20000):
    q, k, v = wl.decode_inputs(wl.DecodeShape('s', 6, 1, 32, 8, 128, T, 'f32', 'f16'))
    qd, kd, vd = (torch.from_numpy(x[0]).cuda() for x in (q, k, v))
    o = torch.empty(32, 128, device='cuda')
    assert lib.attention_launch(o.data_ptr(), qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), T, stream) == 0
    bits = C.c_uint32(7)
    assert lib.attention_status(C.byref(bits), 0, stream) == 0 and bits.value == 0, bits.value
    a, r = wl.error_metrics(o.cpu().numpy(), oracle.best().attn_decode(q, k, v)[0])
    assert a <= wl.ABS_TOL and r <= wl.REL_TOL, (a, r)
print('ok')
"""
    import os
    env = dict(os.environ, LLM_INFER_ATTN_LIB=lib)
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stdout + res.stderr


def test_max_ctas_limits_split_without_changing_result(attention, wl, checker):
    from gpu_util import check_close, run_decode
    q, k, v = _rand(wl, 15, 1, 32, 8, 128, 5000)
    want = checker.attn_decode(q, k, v)
    for cap in (1, 2, 7, 148, 0):
        check_close(wl, run_decode(attention, q, k, v, max_ctas=cap), want, f"max_ctas={cap}")


@pytest.mark.parametrize("H,Hkv,D", [(8, 8, 128), (21, 3, 64), (64, 8, 128), (16, 2, 64), (18, 2, 128)])
@pytest.mark.parametrize("q_dtype,kv_dtype", [("f32", "f16"), ("f16", "f16"), ("f32", "bf16")])
def test_residuals_in_the_idle_rows_against_products_of_their_own(attention, wl, H, Hkv, D, q_dtype, kv_dtype):
    """Up to eight heads per kv head the residual products take the MMAs' rows 8-15; in a generation step (kv_early, lengths
    on the device, prepared output) and with more heads they are products of their own. Same sums in another order: fp32
    rounding (2^-24 each, a few hundred), bf16 probabilities and residuals (2^-17), and the prepared form's 2^-21."""
    import torch
    from gpu_util import to_device
    q, k, v = _rand(wl, H + D, 3, H, Hkv, D, 777, q_dtype, kv_dtype)
    qd, kd, vd = to_device(q, q_dtype), to_device(k, kv_dtype), to_device(v, kv_dtype)
    lens = torch.tensor([777, 16, 500], dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(3, H, Hkv, D)
    rows = attention.attn_decode(qd, kd, vd, lens, workspace=ws, max_ctas=148).double()
    words = torch.empty((3, H, D), dtype=torch.int32, device="cuda")
    attention.attn_decode(qd, kd, vd, lens, out=words, workspace=ws, kv_early=True)
    # words {hi(x0,x1), hi(x2,x3), lo(x0,x1), lo(x2,x3)} of four elements
    h = words.view(torch.float16).view(3, H, D // 4, 2, 4).double()
    own = (h[..., 0, :] + h[..., 1, :]).reshape(3, H, D)
    assert float((rows - own).abs().max()) <= 3e-5 * float(rows.pow(2).mean().sqrt()) + 2.0 ** -21 * float(rows.abs().max())
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("H,Hkv,D", [(8, 8, 128), (21, 3, 64), (64, 8, 128), (16, 2, 64), (18, 2, 128)])
@pytest.mark.parametrize("q_dtype,kv_dtype", [("f32", "f16"), ("f16", "f16"), ("f32", "bf16")])
def test_residuals_in_the_idle_rows_against_two_pass(attention, wl, H, Hkv, D, q_dtype, kv_dtype):
    """Up to eight heads per kv head the residual products take the MMAs' rows 8-15; with two_pass and with more heads they are
    products of their own. Same sums in another order: fp32 rounding (2^-24 each, a few hundred) and bf16 probabilities and
    residuals (2^-17)."""
    import torch
    from gpu_util import to_device
    q, k, v = _rand(wl, H + D, 3, H, Hkv, D, 777, q_dtype, kv_dtype)
    qd, kd, vd = to_device(q, q_dtype), to_device(k, kv_dtype), to_device(v, kv_dtype)
    lens = torch.tensor([777, 16, 500], dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(3, H, Hkv, D)
    rows = attention.attn_decode(qd, kd, vd, lens, workspace=ws, max_ctas=148).double()
    own = attention.attn_decode(qd, kd, vd, lens, workspace=ws, two_pass=True).double()
    assert float((rows - own).abs().max()) <= 3e-5 * float(rows.pow(2).mean().sqrt())
    assert int(ws.status.item()) == 0


@pytest.mark.parametrize("two_pass", [False, True])
@pytest.mark.parametrize("H,Hkv,D,T,lens", [(32, 8, 128, 700, [700, 33, 257]), (32, 8, 128, 40000, [40000, 5, 12345]),
                                            (8, 2, 64, 300, [1, 300, 0]), (18, 2, 128, 333, [333, 17, 48])])
def test_neither_the_early_start_nor_the_output_type_changes_the_sums(attention, wl, H, Hkv, D, T, lens, two_pass):
    """kv_early and the type of the result are no part of the choice between the forms: fp32 results are equal bit for bit, and
    prepared words are the exact split of them. (Short contexts take the clusters, long ones and two_pass the two launches.)"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(H + T)
    q = torch.randn((3, H, D), generator=g, device="cuda")
    k, v = (torch.randn((3, T, Hkv, D), generator=g, device="cuda").half() for _ in range(2))
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    ws = attention.DecodeWorkspace(3, H, Hkv, D)
    plain = attention.attn_decode(q, k, v, kv_len, workspace=ws, two_pass=two_pass)
    x = plain.clamp(-65504, 65504)
    hi = x.half()
    lo = (x - hi.float()).half()
    pairs = torch.stack([t.view(torch.int16).view(3, H, D // 4, 4) for t in (hi, lo)], dim=3)  # four values, then their residuals
    want = pairs.contiguous().view(torch.int32).view(3, H, D)
    for early in (False, True):
        words = torch.empty((3, H, D), dtype=torch.int32, device="cuda")
        attention.attn_decode(q, k, v, kv_len, out=words, workspace=ws, kv_early=early, two_pass=two_pass)
        assert torch.equal(words, want), early
    assert torch.equal(attention.attn_decode(q, k, v, kv_len, workspace=ws, kv_early=True, two_pass=two_pass), plain)
    assert int(ws.status.item()) == 0


# One launch of clusters against the split pass and its merge (which a stated number of CTAs keeps): one to eight kv heads per
# CTA, clusters of one to eight, sub-tiles shared by several warps, CTAs without a tile, empty sequences, odd query groups,
# and NaN in the caches behind the valid rows.
@pytest.mark.parametrize("B,H,Hkv,D,T,lens", [
    (1, 32, 8, 128, 1, None), (1, 32, 4, 64, 512, None), (1, 8, 1, 128, 700, None), (2, 10, 5, 128, 333, [333, 0]),
    (3, 21, 7, 64, 1111, [1, 1111, 64]), (6, 32, 8, 128, 1500, [374, 1499, 17, 1500, 0, 128]), (8, 16, 16, 64, 1000, None),
    (8, 64, 8, 128, 700, [700, 1, 15, 16, 17, 333, 699, 32]), (12, 24, 12, 128, 129, None), (16, 32, 8, 128, 300, None),
    (16, 32, 8, 128, 2100, None)])
@pytest.mark.parametrize("q_dtype,kv_dtype,out", [("f32", "f16", "float32"), ("f16", "f16", "float16"), ("f32", "bf16", "bfloat16")])
def test_cluster_form_against_the_split_form(attention, wl, B, H, Hkv, D, T, lens, q_dtype, kv_dtype, out):
    import torch
    from gpu_util import to_device
    q, k, v = _rand(wl, B * 100 + H + T, B, H, Hkv, D, T, q_dtype, kv_dtype)
    qd, kd, vd = to_device(q, q_dtype), to_device(k, kv_dtype), to_device(v, kv_dtype)
    kv_len = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    for b, n in enumerate(lens or []):
        kd[b, n:], vd[b, n:] = float("nan"), float("nan")
    ws = attention.DecodeWorkspace(B, H, Hkv, D)
    got, launches = [], []
    for cap in (148, 0):
        o = torch.empty((B, H, D), dtype=getattr(torch, out), device="cuda")
        lse = torch.full((B, H), float("nan"), device="cuda")
        before = attention.kernel_launch_count()
        attention.attn_decode(qd, kd, vd, kv_len, out=o, lse=lse, workspace=ws, max_ctas=cap)
        launches.append(attention.kernel_launch_count() - before)
        got.append((o.double(), lse.double()))
    assert launches == [2, 1]
    (o0, l0), (o1, l1) = got
    # fp32 sums in another order (2^-24 per addition, a few hundred of them at most), bf16 probabilities and residuals (2^-17),
    # then the output type's own rounding
    rms = float(o0.pow(2).mean().sqrt()) + 1e-30
    step = {"float32": 0.0, "float16": 2.0 ** -10, "bfloat16": 2.0 ** -7}[out]
    assert float((o0 - o1).abs().max()) <= 3e-5 * rms + step * float(o0.abs().max())
    finite = torch.isfinite(l0)
    assert torch.equal(finite, torch.isfinite(l1)) and float((l0 - l1)[finite].abs().max()) <= 2e-5
    for b, n in enumerate(lens or []):
        assert n > 0 or (bool((o1[b] == 0).all()) and bool(torch.isneginf(l1[b]).all()))
    assert int(ws.status.item()) == 0


# (caches, heads, kv heads, head_dim, rows of a cache): launches. One full cache among short ones keeps most of a cluster launch's
# SMs idle: clusters are taken where that costs less than the second launch, whatever the lengths turn out to be.
@pytest.mark.parametrize("B,H,Hkv,D,cap,launches", [
    (1, 32, 8, 128, 4096, 1), (8, 32, 8, 128, 1024, 1), (16, 32, 8, 128, 512, 1), (16, 32, 4, 64, 2048, 1), (8, 8, 1, 128, 8192, 1),
    (7, 32, 8, 128, 4096, 2), (16, 32, 8, 128, 2048, 2), (16, 32, 8, 128, 4096, 2), (32, 32, 8, 128, 4096, 2), (8, 16, 16, 64, 3000, 2),
    (24, 32, 4, 64, 16384, 2)])
def test_ragged_batches_take_the_clusters_only_where_no_filling_costs_more(attention, B, H, Hkv, D, cap, launches):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line lies elsewhere with another number of SMs")
    cache = torch.zeros((B, cap, Hkv, D), dtype=torch.float16, device="cuda")
    q = torch.zeros((B, H, D), dtype=torch.float16, device="cuda")
    lens = torch.full((B,), 100, dtype=torch.int32, device="cuda")
    before = attention.kernel_launch_count()
    out = attention.attn_decode(q, cache, cache, lens)
    assert attention.kernel_launch_count() - before == launches
    assert bool((out == 0).all())


@pytest.mark.parametrize("H,Hkv,D", [(32, 8, 128), (12, 2, 128), (16, 4, 64), (7, 1, 64)])
@pytest.mark.parametrize("q_dtype,kv_dtype", [("f16", "f16"), ("f32", "bf16")])
def test_a_stated_capacity_is_no_promise_of_readable_rows(attention, pkg, wl, H, Hkv, D, q_dtype, kv_dtype):
    """kv_capacity bounds the lengths and nothing else: here it is stated larger than the distance between two sequences, whose
    last one ends with the memory itself, and the row pitch is wider than a row. A sequence's last tile is moved back to end
    with the sequence: fewer rows than a tile, exactly one, one more, and remainders around the 16 rows of a warp."""
    import ctypes as C

    import torch
    from gpu_util import to_device
    T, spare, lib = 257, 8, pkg.binding.load()
    for lens in ([257, 1, 128, 17], [256, 16, 129, 2], [15, 255, 0, 127], [3, 5, 9, 257]):
        B = len(lens)
        q, k, v = _rand(wl, H + lens[0], B, H, Hkv, D, T, q_dtype, kv_dtype)
        qd, kd, vd = to_device(q, q_dtype), to_device(k, kv_dtype), to_device(v, kv_dtype)
        pitch = Hkv * D + spare
        flat = [torch.full((((B - 1) * T + lens[-1] - 1) * pitch + Hkv * D,), float("nan"), dtype=kd.dtype, device="cuda")
                for _ in range(2)]
        for buf, cache in zip(flat, (kd, vd)):
            for b, n in enumerate(lens):
                for i in range(n):
                    buf[(b * T + i) * pitch:][:Hkv * D] = cache[b, i].reshape(-1)
        kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
        ws = attention.DecodeWorkspace(B, H, Hkv, D)
        got = []
        for two_pass in (1, 0):
            a, out, _, _ = attention._decode_args(qd, kd, vd, kv_len, None, None, torch.float32, 0.0, ws, 0)
            a.k, a.v, a.kv_row_stride, a.kv_batch_stride = flat[0].data_ptr(), flat[1].data_ptr(), pitch, T * pitch
            a.kv_capacity, a.two_pass = 600, two_pass
            before = attention.kernel_launch_count()
            assert lib.attn_decode(C.byref(a), torch.cuda.current_stream().cuda_stream) == 0
            assert attention.kernel_launch_count() - before == 1 + two_pass
            got.append(out.double())
        rms = float(got[0].pow(2).mean().sqrt())
        assert float((got[0] - got[1]).abs().max()) <= 3e-5 * rms  # another order of the sums, as in the test above
        assert int(ws.status.item()) == 0


def test_merge_entry_point(attention, wl, port):
    import torch
    q, k, v = wl.decode_inputs(wl.C4, kv_len=999)
    want, part_o, part_lse = port.attn_decode_sharded(q.astype(np.float32)[0], k[0], v[0], 5)
    part_lse[3] = -np.inf  # an empty shard
    want = np.stack([port.lse_merge(part_o[:, h], part_lse[:, h])[0] for h in range(32)])
    lse = torch.empty(32, dtype=torch.float32, device="cuda")
    got = attention.attn_merge(torch.from_numpy(part_o).cuda(), torch.from_numpy(part_lse).cuda(), lse=lse)
    torch.cuda.synchronize()
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=0, atol=1e-5)
    all_empty = torch.full((3, 8), float("-inf"), device="cuda")
    z = attention.attn_merge(torch.randn(3, 8, 128, device="cuda"), all_empty)
    assert torch.equal(z, torch.zeros_like(z))


@pytest.mark.parametrize("n_parts", [1, 7, 24, 25, 49, 97, 148, 301])
@pytest.mark.parametrize("D", [64, 128])
def test_merge_of_many_partials(attention, port, n_parts, D):
    """From one to a few hundred partials per row (a single long sequence leaves one per split-pass CTA): same result
    as the restated LSE merge, empty partials (lse = -inf) included."""
    import torch
    rng = np.random.default_rng(n_parts * 7 + D)
    rows = 5
    part_o = rng.standard_normal((n_parts, rows, D), dtype=np.float32)
    part_lse = (rng.standard_normal((n_parts, rows), dtype=np.float32) * 3).astype(np.float32)
    part_lse[rng.random((n_parts, rows)) < 0.2] = -np.inf
    part_lse[:, 4] = -np.inf  # a row with nothing at all
    lse = torch.empty(rows, dtype=torch.float32, device="cuda")
    got = attention.attn_merge(torch.from_numpy(part_o).cuda(), torch.from_numpy(part_lse).cuda(), lse=lse)
    torch.cuda.synchronize()
    got, lse = got.cpu().numpy(), lse.cpu().numpy()
    for r in range(rows):
        want, want_lse = port.lse_merge(part_o[:, r], part_lse[:, r])
        if np.isinf(part_lse[:, r]).all():
            assert (got[r] == 0).all() and lse[r] == -np.inf
        else:
            np.testing.assert_allclose(got[r], want, rtol=0, atol=2e-5)
            assert abs(lse[r] - want_lse) <= 1e-5 * max(1.0, abs(want_lse))


@pytest.mark.parametrize("n_parts", [1, 5, 6, 7, 16])
@pytest.mark.parametrize("D", [32, 64, 128, 256])
def test_merge_of_many_rows_with_few_partials(attention, port, n_parts, D):
    """Hundreds of rows with a handful of partials each (batched decode) take the warp-per-row form of the merge pass:
    same result as the restated LSE merge, empty partials and empty rows included."""
    import torch
    rng = np.random.default_rng(n_parts * 11 + D)
    rows = 300
    part_o = rng.standard_normal((n_parts, rows, D), dtype=np.float32)
    part_lse = (rng.standard_normal((n_parts, rows), dtype=np.float32) * 3).astype(np.float32)
    part_lse[rng.random((n_parts, rows)) < 0.2] = -np.inf
    part_lse[:, 7] = -np.inf
    lse = torch.empty(rows, dtype=torch.float32, device="cuda")
    got = attention.attn_merge(torch.from_numpy(part_o).cuda(), torch.from_numpy(part_lse).cuda(), lse=lse)
    torch.cuda.synchronize()
    got, lse = got.cpu().numpy(), lse.cpu().numpy()
    for r in range(0, rows, 13):
        want, want_lse = port.lse_merge(part_o[:, r], part_lse[:, r])
        if np.isinf(part_lse[:, r]).all():
            assert (got[r] == 0).all() and lse[r] == -np.inf
        else:
            np.testing.assert_allclose(got[r], want, rtol=0, atol=2e-5)
            assert abs(lse[r] - want_lse) <= 1e-5 * max(1.0, abs(want_lse))
    assert (got[7] == 0).all() and lse[7] == -np.inf


def _sharded_single_gpu(attention, q, k, v, world, rank, bufs, out, status_ws, step=0, poll_limit=0):
    import torch
    return attention.attn_decode_sharded(q, k, v, peer_buffers=[b.data_ptr() for b in bufs], world_size=world,
                                         rank=rank, step=step, poll_limit=poll_limit, out=out, workspace=status_ws)


def test_fused_exchange_with_one_rank_equals_plain_decode(attention, wl, checker):
    """World size 1: the exchange path (peer stores, flags, wait, cross merge) runs against the rank's own buffer."""
    import torch
    from gpu_util import check_close, to_device
    q, k, v = _rand(wl, 41, 2, 32, 8, 128, 3000, "f16", "f16")
    qd, kd, vd = to_device(q, "f16"), to_device(k, "f16"), to_device(v, "f16")
    ws = attention.DecodeWorkspace(2, 32, 8, 128)
    buf = torch.zeros(attention.exchange_bytes(2, 32, 128, 1) // 4, device="cuda")
    want = checker.attn_decode(q.astype(np.float32), k, v)
    for call in range(3):  # consecutive steps alternate the record parity and advance the device-side step counter
        out = torch.full((2, 32, 128), float("nan"), device="cuda")
        _sharded_single_gpu(attention, qd, kd, vd, 1, 0, [buf], out, ws)
        torch.cuda.synchronize()
        check_close(wl, out.cpu().numpy(), want, f"fused exchange, call {call}")
    assert int(ws.status.item()) == 0
    ctl = buf.view(torch.int64)[-2:].tolist()
    assert ctl == [3, 0]  # three steps completed, no cell pending


def test_fused_exchange_times_out_cleanly_when_a_peer_never_arrives(attention, wl, checker):
    """World size 2 with nobody playing rank 1: the wait on rank 1's flags must run out, set the status bit and leave
    the output untouched; the context stays usable (a normal decode works right after)."""
    import torch
    from gpu_util import check_close, to_device
    q, k, v = _rand(wl, 42, 1, 32, 8, 128, 500, "f16", "f16")
    qd, kd, vd = to_device(q, "f16"), to_device(k, "f16"), to_device(v, "f16")
    ws = attention.DecodeWorkspace(1, 32, 8, 128)
    n = attention.exchange_bytes(1, 32, 128, 2) // 4
    mine, absent_peer = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    out = torch.full((1, 32, 128), float("nan"), device="cuda")
    _sharded_single_gpu(attention, qd, kd, vd, 2, 0, [mine, absent_peer], out, ws, step=1, poll_limit=200)
    torch.cuda.synchronize()
    assert int(ws.status.item()) & 1  # ATTN_STATUS_WAIT_TIMEOUT
    assert torch.isnan(out).all()
    # this rank's record did reach the "peer": what a live rank 1 would have merged (step 1 -> parity 1, source rank 0)
    rec_o, rec_lse, steps = attention.exchange_record(absent_peer, 1, 32, 128, 2, parity=1, source_rank=0)
    assert (steps == 1).all()
    want = checker.attn_decode(q.astype(np.float32), k, v)
    check_close(wl, rec_o.view(1, 32, 128).cpu().numpy(), want, "record delivered to the peer buffer")
    assert torch.isfinite(rec_lse).all()
    ws.status.zero_()
    got = attention.attn_decode(qd, kd, vd, workspace=ws)
    torch.cuda.synchronize()
    check_close(wl, got.cpu().numpy(), want, "decode after a timed-out exchange")
    assert int(ws.status.item()) == 0


def test_host_threads_with_calls_of_different_sizes(attention, pkg):
    """Three threads, each with its own stream and workspace, whose calls take the same kernel with different amounts of shared
    memory (4 to 32 KB of query rows): no launch is refused and every result stays the thread's own."""
    import ctypes as C
    import threading

    import torch
    lib, errors = pkg.binding.load(), []

    def worker(H, max_ctas, start):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                g = torch.Generator(device="cuda").manual_seed(H)
                q = torch.randn((1, H, 128), generator=g, device="cuda").half()
                k, v = (torch.randn((1, 64, 8, 128), generator=g, device="cuda").half() for _ in range(2))
                ws = attention.DecodeWorkspace(1, H, 8, 128)
                first = attention.attn_decode(q, k, v, workspace=ws, max_ctas=max_ctas)
                args, out, _, _ = attention._decode_args(q, k, v, None, torch.empty_like(first), None, None, 0.0, ws, max_ctas)
                ref, raw, call = C.byref(args), stream.cuda_stream, lib.attn_decode
                start.wait()
                codes = {call(ref, raw) for _ in range(20000)}
                stream.synchronize()
                assert codes == {0}, codes
                assert torch.equal(out, first) and int(ws.status.item()) == 0
        except Exception as e:  # noqa: BLE001 (reported by the test's thread)
            errors.append(e)

    for max_ctas in (148, 0):
        start = threading.Barrier(3, timeout=60)
        threads = [threading.Thread(target=worker, args=(H, max_ctas, start)) for H in (8, 64, 32)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
