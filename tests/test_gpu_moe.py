"""GPU parity of the mixture-of-experts steps around the grouped GEMM: block alignment (bit-exact against
the reference's stored outputs and the oracle), row gather (bit-exact), silu_and_mul (the reference's
tolerance), the fused silu_and_mul + MXFP4 quantisation, the weighted combine, and the whole expert MLP.
Mirrors tests/kernel/moe/moe_align_block_size_test.py and tests/kernel/moe_test.py of the reference."""

import numpy as np
import pytest
import torch

import wave_b200 as wb
from conftest import GOLDEN
from oracle import moe_oracle
from oracle import mxfp4_oracle as orc
from wave_b200 import moe, ops
from wave_b200.grouped import ExpertWeights

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run_align(topk_ids, experts, block, with_inverse=True):
    n = topk_ids.numel()
    cap = n + experts * (block - 1)
    sorted_ids = torch.empty(cap, dtype=torch.int32, device=DEV)
    expert_ids = torch.full((-(cap // -block),), -1, dtype=torch.int32, device=DEV)
    post = torch.empty(1, dtype=torch.int32, device=DEV)
    inverse = torch.empty(n, dtype=torch.int32, device=DEV) if with_inverse else None
    wb.moe_align_block_size(topk_ids.to(DEV), experts, block, sorted_ids, expert_ids, post, inverse)
    return sorted_ids.cpu().numpy(), expert_ids.cpu().numpy(), int(post.item()), None if inverse is None else inverse.cpu().numpy()


def test_moe_align_block_size_golden():
    g = np.load(GOLDEN / "moe_align.npz")
    ci = 0
    while f"case{ci}_params" in g.files:
        tokens, topk, block, experts = (int(v) for v in g[f"case{ci}_params"])
        ids = torch.from_numpy(g[f"case{ci}_topk_ids"])
        sorted_ids, expert_ids, post, inverse = run_align(ids, experts, block)
        assert post == int(g[f"case{ci}_post_pad"][0])
        assert np.array_equal(sorted_ids, g[f"case{ci}_sorted_ids"])
        assert np.array_equal(expert_ids, g[f"case{ci}_expert_ids"])
        assert np.array_equal(sorted_ids[inverse], np.arange(tokens * topk))
        ci += 1
    assert ci >= 6


@pytest.mark.parametrize("num_tokens", [1, 33, 256, 4096])
@pytest.mark.parametrize("block_size", [16, 32, 64, 128])
@pytest.mark.parametrize("num_experts", [4, 8, 64, 256])
def test_moe_align_block_size_matches_oracle(num_tokens, block_size, num_experts):
    """The reference test's sweep (moe_align_block_size_test.py:14-17), widened; int32 and int64 ids."""
    g = torch.Generator().manual_seed(num_tokens * 7 + block_size + num_experts)
    _, topk_ids = torch.topk(torch.rand(num_tokens, num_experts, generator=g), k=2, dim=1)
    exp = moe_oracle.moe_align_block_size(topk_ids.numpy(), num_experts, block_size,
                                          topk_ids.numel() + num_experts * (block_size - 1),
                                          -((topk_ids.numel() + num_experts * (block_size - 1)) // -block_size))
    for ids in (topk_ids, topk_ids.to(torch.int32)):
        sorted_ids, expert_ids, post, inverse = run_align(ids, num_experts, block_size)
        assert post == exp[2] and post % block_size == 0
        assert np.array_equal(sorted_ids, exp[0]) and np.array_equal(expert_ids, exp[1]) and np.array_equal(inverse, exp[3])


def test_moe_align_block_size_skewed_and_empty():
    ids = torch.full((1000, 2), 3, dtype=torch.int64)  # every pair on one expert, all others empty
    exp = moe_oracle.moe_align_block_size(ids.numpy(), 8, 128, 2000 + 8 * 127, -((2000 + 8 * 127) // -128))
    sorted_ids, expert_ids, post, inverse = run_align(ids, 8, 128)
    assert post == 2048 and np.array_equal(sorted_ids, exp[0]) and np.array_equal(expert_ids, exp[1])
    with pytest.raises(ValueError):  # outputs too small for the worst case
        wb.moe_align_block_size(ids.to(DEV), 8, 128, torch.empty(2000, dtype=torch.int32, device=DEV),
                                torch.empty(30, dtype=torch.int32, device=DEV), torch.empty(1, dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("row_bytes", [256, 8, 100])
def test_gather_rows_bit_exact(row_bytes):
    g = torch.Generator().manual_seed(row_bytes)
    src = torch.randint(0, 256, (50, row_bytes), dtype=torch.uint8, generator=g)
    _, ids = torch.topk(torch.rand(50, 8, generator=g), k=2, dim=1)
    sorted_ids, _, post, _ = run_align(ids, 8, 16, with_inverse=False)
    out = torch.full((post, row_bytes), 0xAB, dtype=torch.uint8, device=DEV)
    moe.gather_rows(src.to(DEV), torch.from_numpy(sorted_ids).to(DEV), 100, 2, out)
    exp = torch.zeros(post, row_bytes, dtype=torch.uint8)
    real = torch.from_numpy(sorted_ids[:post]) < 100
    exp[real] = src[torch.from_numpy(sorted_ids[:post])[real].long() // 2]
    assert torch.equal(out.cpu(), exp)


@pytest.mark.parametrize("m,n", [(1, 128), (33, 1024), (64, 200), (5, 30)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_silu_and_mul_as_the_reference_tests_it(m, n, dtype):
    """get_wave_silu_and_mul_kernel / silu_and_mul of tests/kernel/moe_test.py:43-79 (rtol 1e-1, atol 1e-2 there)."""
    kernel, symbols = wb.get_silu_and_mul_kernel(m, n, dtype)
    silu = wb.wave_compile(wb.WaveCompileOptions(subs=symbols, canonicalize=True, schedule=wb.SchedulingType.NONE), kernel)
    g = torch.Generator().manual_seed(m + n)
    gate = torch.randn(m, n, generator=g).to(dtype)
    up = torch.randn(m, n, generator=g).to(dtype)
    out = torch.zeros(m, n, dtype=dtype, device=DEV)
    silu(gate.to(DEV), up.to(DEV), out)
    ref = moe_oracle.silu_and_mul(gate, up)
    torch.testing.assert_close(out.cpu().float(), ref, rtol=1e-1, atol=1e-2)
    # and much tighter: the kernel's fast exponential and division are good to ~1e-6 relative, then one
    # rounding to the output type
    if dtype == torch.float32:
        torch.testing.assert_close(out.cpu(), ref, rtol=1e-5, atol=1e-6)
    else:
        assert int(orc.bf16_ulp_distance(out, ref).max()) <= 1


def test_silu_and_mul_on_column_halves_with_fused_quantisation():
    rows, inter = 300, 512
    g = torch.Generator().manual_seed(3)
    h = (torch.randn(rows, 2 * inter, generator=g) * 2).to(torch.bfloat16)
    hd = h.to(DEV)
    out, q, s = wb.silu_and_mul(hd[:, :inter], hd[:, inter:], out=torch.empty(rows, inter, dtype=torch.bfloat16, device=DEV),
                                quantize=True)
    ref = moe_oracle.silu_and_mul(h[:, :inter], h[:, inter:])
    assert int(orc.bf16_ulp_distance(out, ref).max()) <= 1
    # The codes come from the kernel's own f32 values, which differ from the oracle's by a few ulps, so a value
    # next to a rounding boundary may land on the neighbouring code: nearly all codes and scales are those of the
    # oracle's quantiser, and every dequantised value is within the quantiser's worst-case error of the reference
    # (2 units of the block's scale: values between 6 and 8 units are clamped to 6).
    q_ref, s_ref = orc.quantize_mxfp4(ref)
    assert float((s.cpu() != s_ref).float().mean()) < 1e-3
    qc, qr = q.cpu(), q_ref
    nib_diff = ((qc & 0xF) != (qr & 0xF)).float().mean() + ((qc >> 4) != (qr >> 4)).float().mean()
    assert float(nib_diff) < 2e-3
    deq = orc.dequant_mxfp4(qc, s.cpu())
    unit = orc.e8m0_to_f32(s.cpu().float()).repeat_interleave(32, dim=1)
    assert bool(((deq - ref).abs() <= unit * 2.0 + 1e-6).all())
    # quantise-only form gives the same codes
    _, q2, s2 = wb.silu_and_mul(hd[:, :inter], hd[:, inter:], quantize=True)
    assert torch.equal(q, q2) and torch.equal(s, s2)


def test_combine_matches_weighted_sum():
    T, k, cols = 77, 2, 200
    g = torch.Generator().manual_seed(9)
    y = torch.randn(300, cols, generator=g).to(torch.bfloat16)
    row_of = torch.randint(0, 300, (T * k,), generator=g, dtype=torch.int32)
    row_of[5] = -1
    w = torch.rand(T * k, generator=g)
    out = torch.empty(T, cols, dtype=torch.bfloat16, device=DEV)
    moe.combine(y.to(DEV), row_of.to(DEV), w.to(DEV), k, out)
    contrib = torch.where((row_of >= 0).view(-1, 1), w.view(-1, 1) * y.float()[row_of.clamp(min=0).long()], torch.zeros(1))
    ref = contrib.view(T, k, cols).sum(1)
    assert int(orc.bf16_ulp_distance(out, ref).max()) <= 1


@pytest.mark.parametrize("T,E,K,inter", [(33, 8, 512, 256), (256, 4, 1024, 512), (1, 8, 256, 128)])
def test_expert_mlp_against_oracle(T, E, K, inter):
    """Whole MXFP4 expert MLP against the oracle's expert loop (torch_ref_moe's structure). Tolerance: the
    reference's own MoE tolerance (rtol 1e-1, atol 1e-2, tests/kernel/moe_test.py:258), which absorbs the
    re-quantisation of hidden activations whose f32 values differ from the oracle's in the last bits."""
    g = torch.Generator().manual_seed(T + E)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    logits = torch.randn(T, E, generator=g)
    w1, w1s, w2, w2s = [], [], [], []
    for e in range(E):
        q, s = orc.quantize_mxfp4(torch.randn(2 * inter, K, generator=g) * 0.05)
        w1.append(q); w1s.append(s)
        q, s = orc.quantize_mxfp4(torch.randn(K, inter, generator=g) * 0.05)
        w2.append(q); w2s.append(s)
    mlp = wb.MXFP4ExpertMLP([t.to(DEV) for t in w1], [t.to(DEV) for t in w1s], [t.to(DEV) for t in w2],
                            [t.to(DEV) for t in w2s], top_k=2)
    out = mlp(x.to(DEV), logits.to(DEV))
    ref = moe_oracle.expert_mlp(x, w1, w1s, w2, w2s, logits, 2)
    torch.testing.assert_close(out.cpu().float(), ref, rtol=1e-1, atol=1e-2)
    # and relative to the output's own scale: mean error well under one percent of the rms
    rel = (out.cpu().float() - ref).abs().mean() / ref.pow(2).mean().sqrt()
    assert float(rel) < 2e-2
    ops.check_device_status()


def test_device_driven_grouped_gemm_matches_host_offsets_form():
    """wb200_mxfp4_moe_gemm (routing read from the alignment kernel's device outputs) against
    wb200_mxfp4_grouped_gemm (row offsets given by the host) on the same routed rows: identical bits."""
    from wave_b200.grouped import ExpertWeights, grouped_scaled_gemm, moe_scaled_gemm
    T, E, K, N, k = 700, 5, 512, 384, 2
    g = torch.Generator().manual_seed(21)
    _, ids = torch.topk(torch.rand(T, E, generator=g), k=k, dim=1)
    ids[:, :] = torch.where(ids == 3, torch.zeros_like(ids), ids)  # expert 3 gets no rows
    n = T * k
    cap = (n + E * 255 + 255) // 256 * 256
    sorted_ids, expert_ids, post, _ = run_align(ids, E, 256)
    sorted_ids = np.concatenate([sorted_ids, np.full(cap - sorted_ids.size, n, dtype=np.int32)])
    xq = torch.randint(0, 256, (T, K // 2), dtype=torch.uint8, generator=g)
    xs = torch.randint(122, 129, (T, K // 32), dtype=torch.uint8, generator=g)
    w = [torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g) for _ in range(E)]
    ws = [torch.randint(122, 129, (N, K // 32), dtype=torch.uint8, generator=g) for _ in range(E)]
    experts = ExpertWeights([t.to(DEV) for t in w], [t.to(DEV) for t in ws])
    a = torch.empty(cap, K // 2, dtype=torch.uint8, device=DEV)
    a_s = torch.empty(cap, K // 32, dtype=torch.uint8, device=DEV)
    sid = torch.from_numpy(sorted_ids).to(DEV)
    moe.gather_rows(xq.to(DEV), sid, n, k, a)
    moe.gather_rows(xs.to(DEV), sid, n, k, a_s)
    c_dev = torch.full((cap, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    eid = torch.full((cap // 256,), -1, dtype=torch.int32, device=DEV)
    eid[: expert_ids.size] = torch.from_numpy(expert_ids).to(DEV)[: cap // 256]
    moe_scaled_gemm(a, a_s, experts, eid, torch.tensor([post], dtype=torch.int32, device=DEV), c_dev)
    counts = torch.bincount(ids.reshape(-1), minlength=E).tolist()
    offsets = [0]
    for cnt in counts:
        offsets.append(offsets[-1] + (cnt + 255) // 256 * 256)
    assert offsets[-1] == post
    c_host = torch.empty(post, N, dtype=torch.bfloat16, device=DEV)
    grouped_scaled_gemm(a[:post], a_s[:post], experts, offsets, c_host)
    assert torch.equal(c_dev[:post].view(torch.int16), c_host.view(torch.int16))
    assert bool(c_dev[post:].isnan().all())  # row blocks past the padded total are not touched
    # and against the oracle for one expert's rows
    e = 1
    rows = slice(offsets[e], offsets[e] + counts[e])
    ref = orc.scaled_gemm(a[rows].cpu(), a_s[rows].cpu(), w[e], ws[e])
    assert int(orc.bf16_ulp_distance(c_dev[rows], ref).max()) <= 1
    ops.check_device_status()


def test_expert_mlp_forward_can_be_captured_in_a_cuda_graph():
    """No step of the forward pass reads the routing back to the host."""
    T, E, K, inter = 64, 4, 512, 256
    g = torch.Generator().manual_seed(2)
    w1, w1s, w2, w2s = [], [], [], []
    for e in range(E):
        q, s = orc.quantize_mxfp4(torch.randn(2 * inter, K, generator=g) * 0.05)
        w1.append(q.to(DEV)); w1s.append(s.to(DEV))
        q, s = orc.quantize_mxfp4(torch.randn(K, inter, generator=g) * 0.05)
        w2.append(q.to(DEV)); w2s.append(s.to(DEV))
    mlp = wb.MXFP4ExpertMLP(w1, w1s, w2, w2s, top_k=2)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    logits = torch.randn(T, E, generator=g).to(DEV)
    eager = mlp(x, logits)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = mlp(x, logits)
    x.copy_(torch.randn(T, K, generator=g).to(torch.bfloat16))  # new tokens, same buffers
    graph.replay()
    torch.cuda.synchronize()
    again = mlp(x, logits)
    torch.cuda.synchronize()
    assert torch.equal(captured, again) and not torch.equal(captured, eager)
    ops.check_device_status()


def test_quantize_scatter_equals_quantise_then_gather_on_routed_rows():
    T, E, K, k = 300, 6, 1024, 2
    g = torch.Generator().manual_seed(31)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    _, ids = torch.topk(torch.rand(T, E, generator=g), k=k, dim=1)
    sorted_ids, _, post, inverse = run_align(ids, E, 256)
    cap = (T * k + E * 255 + 255) // 256 * 256
    q = torch.full((cap, K // 2), 0xEE, dtype=torch.uint8, device=DEV)
    s = torch.full((cap, K // 32), 0xEE, dtype=torch.uint8, device=DEV)
    moe.quantize_scatter(x.to(DEV), torch.from_numpy(inverse).to(DEV), k, q, s)
    q_ref, s_ref = orc.quantize_mxfp4(x.float())
    routed = torch.from_numpy(sorted_ids[:post]).long()
    real = routed < T * k
    pos = torch.arange(post)[real]
    assert torch.equal(q.cpu()[pos], q_ref[routed[real] // k]) and torch.equal(s.cpu()[pos], s_ref[routed[real] // k])
    untouched = torch.ones(cap, dtype=torch.bool)
    untouched[pos] = False
    assert bool((q.cpu()[untouched] == 0xEE).all()) and bool((s.cpu()[untouched] == 0xEE).all())


def test_silu_and_mul_row_limit_from_device():
    rows, n = 512, 256
    g = torch.Generator().manual_seed(8)
    h = torch.randn(rows, 2 * n, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((rows, n), -3.0, dtype=torch.bfloat16, device=DEV)
    limit = torch.tensor([384], dtype=torch.int32, device=DEV)
    wb.silu_and_mul(h[:, :n], h[:, n:], out=out, num_rows=limit)
    ref = moe_oracle.silu_and_mul(h[:384, :n].cpu(), h[:384, n:].cpu())
    assert int(orc.bf16_ulp_distance(out[:384], ref).max()) <= 1
    assert bool((out[384:] == -3.0).all())


def _poison(nbytes=1 << 28):
    """Leave freed blocks full of 0xFF in the allocator: workspaces then start as NaN scales and saturated codes."""
    blocks = [torch.full((n,), 255, dtype=torch.uint8, device=DEV) for n in (nbytes, 1 << 22, 1 << 20, 1 << 18)]
    torch.cuda.synchronize()
    del blocks


@pytest.mark.parametrize("T,E,K,inter,N,k,x_dtype,l_dtype", [
    (1, 4, 256, 128, 256, 1, torch.bfloat16, torch.float32),      # one token, one atom pair, one block
    (16, 8, 416, 384, 160, 2, torch.float32, torch.bfloat16),     # K, N ragged, odd atom count of the hidden columns
    (17, 3, 1024, 128, 96, 3, torch.bfloat16, torch.float16),     # every expert gets every token
    (64, 32, 512, 256, 512, 8, torch.bfloat16, torch.float32),    # the large table of experts
    (128, 9, 288, 640, 256, 2, torch.bfloat16, torch.float32),    # the largest batch of the decode form
    (129, 9, 288, 640, 256, 2, torch.bfloat16, torch.float32),    # the smallest of the tile form
    (700, 2, 512, 384, 160, 1, torch.float32, torch.float32),
    (513, 17, 1056, 128, 4096, 4, torch.bfloat16, torch.bfloat16),
])
def test_expert_mlp_single_call_form(T, E, K, inter, N, k, x_dtype, l_dtype):
    """The single native call against the oracle and against the step-by-step form, over both row layouts. The hidden codes
    of the two forms are the same; the routing weights may differ in their last bits (another order of the softmax's sum),
    so an output by one rounding to bf16, 2^-8 of itself. Against the oracle the f32 sums in front of the bf16 rounding
    differ in their last bits: a value next to a rounding boundary moves by 2^-8, and about 2^-8 * 8 of those cross one of
    the 4-bit quantiser, by a third of the value. With one in a hundred next to a boundary that is a share of 3e-4,
    a relative 2-norm of sqrt(3e-4) / 3 ~ 6e-3, and 2^-8 / sqrt(3) of bf16 rounding in y and the output: 1.5e-2 in all."""
    g = torch.Generator().manual_seed(T * 31 + E)
    x = torch.randn(T, K, generator=g).to(x_dtype)
    # 16-bit logits drawn at random tie (8 bits of mantissa, 513 rows), and the oracle's top-k breaks ties in another order, which
    # is another, equally correct result: distinct values per row, exact in either type
    logits = torch.randn(T, E, generator=g) if l_dtype == torch.float32 else torch.rand(T, E, generator=g).argsort(1).float() * 0.25
    logits = logits.to(l_dtype)
    w1, w1s, w2, w2s = [], [], [], []
    for e in range(E):
        q, s = orc.quantize_mxfp4(torch.randn(2 * inter, K, generator=g) * 0.05)
        w1.append(q); w1s.append(s)
        q, s = orc.quantize_mxfp4(torch.randn(N, inter, generator=g) * 0.05)
        w2.append(q); w2s.append(s)
    mlp = wb.MXFP4ExpertMLP([t.to(DEV) for t in w1], [t.to(DEV) for t in w1s], [t.to(DEV) for t in w2],
                            [t.to(DEV) for t in w2s], top_k=k)
    xd, ld = x.to(DEV), logits.to(DEV)
    assert mlp._takes_fused(xd, ld)
    _poison()
    out = mlp(xd, ld)
    ref = moe_oracle.expert_mlp(x, w1, w1s, w2, w2s, logits.float(), k)
    assert float((out.cpu().float() - ref).norm() / ref.norm()) < 1.5e-2
    steps = mlp._forward_steps(xd, ld).float()
    assert bool(((out.float() - steps).abs() <= 2 ** -7 * steps.abs() + 1e-6 * steps.abs().max()).all())
    assert torch.equal(mlp(xd, ld), out)  # whichever CTA takes a tile
    wide = torch.zeros(T, K + 64, dtype=x_dtype, device=DEV)
    wide[:, 32:K + 32] = xd
    assert torch.equal(mlp(wide[:, 32:K + 32], ld.t().contiguous().t()), out)  # row pitch of x, column-major logits
    ops.check_device_status()


@pytest.mark.parametrize("T", [40, 200])
def test_expert_mlp_single_call_form_special_logits(T):
    """Masked experts (-inf), ties and a NaN row: the same tokens through the library router and the step-by-step form."""
    E, K, inter, N, k = 6, 256, 128, 128, 2
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    logits = torch.randn(T, E, generator=g)
    logits[3, 1:] = float("-inf")
    logits[4, ::2] = float("-inf")
    logits[5, 2] = float("nan")
    w1 = [orc.quantize_mxfp4(torch.randn(2 * inter, K, generator=g) * 0.05) for _ in range(E)]
    w2 = [orc.quantize_mxfp4(torch.randn(N, inter, generator=g) * 0.05) for _ in range(E)]
    mlp = wb.MXFP4ExpertMLP([q.to(DEV) for q, _ in w1], [s.to(DEV) for _, s in w1], [q.to(DEV) for q, _ in w2],
                            [s.to(DEV) for _, s in w2], top_k=k)
    out = mlp(x, logits.to(DEV)).float()
    steps = mlp._forward_steps(x, logits.to(DEV)).float()
    assert bool(out[5].isnan().all()) and bool(steps[5].isnan().all())
    rows = torch.arange(T, device=DEV) != 5
    assert bool(((out[rows] - steps[rows]).abs() <= 2 ** -7 * steps[rows].abs() + 1e-6 * steps[rows].abs().max()).all())
    # a tie between all experts: any of them is a correct choice; the lower ones are taken
    tied = torch.zeros(T, E, device=DEV)
    first = torch.full((T, E), -30.0, device=DEV)
    first[:, :k] = 0.0
    torch.testing.assert_close(mlp(x, tied).float() * 3.0, mlp(x, first).float(), rtol=2 ** -7, atol=1e-6)
    ops.check_device_status()


def _small_expert_mlp(seed, E=4, K=256, inter=128, N=96, k=2):
    g = torch.Generator().manual_seed(seed)
    w1 = [orc.quantize_mxfp4(torch.randn(2 * inter, K, generator=g) * 0.05) for _ in range(E)]
    w2 = [orc.quantize_mxfp4(torch.randn(N, inter, generator=g) * 0.05) for _ in range(E)]
    mlp = wb.MXFP4ExpertMLP([q.to(DEV) for q, _ in w1], [s.to(DEV) for _, s in w1], [q.to(DEV) for q, _ in w2], [s.to(DEV) for _, s in w2],
                            top_k=k)
    return w1, w2, mlp


@pytest.mark.parametrize("T", [1, 16, 128, 200])
@pytest.mark.parametrize("how", ["object", "in place", "in place under a graph"])
def test_expert_mlp_reads_the_weights_as_they_are_at_the_call(T, how):
    """Weights replaced between two calls, as another object, in place, and in place between the capture and the replay of a
    graph: the second result is that of the new weights (other codes and other scales), at decode and prefill sizes.
    Tolerance as in test_expert_mlp_single_call_form."""
    k = 2
    _, w2, mlp = _small_expert_mlp(1, k=k)
    new = [(q, s + 2) for q, s in _small_expert_mlp(2, k=k)[0]]
    g = torch.Generator().manual_seed(3)
    x, logits = torch.randn(T, mlp.K, generator=g).to(torch.bfloat16), torch.randn(T, mlp.E, generator=g)
    xd, ld = x.to(DEV), logits.to(DEV)
    mlp(xd, ld)
    if how.endswith("graph"):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = mlp(xd, ld)
    if how == "object":
        mlp.w1 = ExpertWeights([q.to(DEV) for q, _ in new], [s.to(DEV) for _, s in new])
    else:
        for e, (q, s) in enumerate(new):
            mlp.w1.b[e].copy_(q)
            ops.repack_scales(s.to(DEV), out=mlp.w1.b_sf[e].data)
    if how.endswith("graph"):
        graph.replay()
    else:
        out = mlp(xd, ld)
    ref = moe_oracle.expert_mlp(x, [q for q, _ in new], [s for _, s in new], [q for q, _ in w2], [s for _, s in w2], logits, k)
    assert float((out.cpu().float() - ref).norm() / ref.norm()) < 1.5e-2
    ops.check_device_status()


@pytest.mark.parametrize("T", [16, 200])
@pytest.mark.parametrize("where", ["instance", "subclass", "class"])
def test_expert_mlp_calls_the_router_it_was_given(T, where, monkeypatch):
    """A `route` of the caller's own, wherever it was set, decides the experts: negated logits through the library's router
    give the result of the same logits through a router that negates them. Both sides run the same GEMMs on the same codes;
    the weights may differ in the last bits of the softmax, an output by one rounding to bf16."""
    mlp = _small_expert_mlp(1)[2]
    g = torch.Generator().manual_seed(T)
    x, logits = torch.randn(T, mlp.K, generator=g).to(torch.bfloat16).to(DEV), torch.randn(T, mlp.E, generator=g).to(DEV)
    expected = mlp(x, -logits).float()
    library = wb.MXFP4ExpertMLP.route
    if where == "instance":
        mlp.route = lambda r: library(mlp, -r)
    elif where == "subclass":
        mlp.__class__ = type("Routed", (wb.MXFP4ExpertMLP,), {"route": lambda self, r: library(self, -r)})
    else:
        monkeypatch.setattr(wb.MXFP4ExpertMLP, "route", lambda self, r: library(self, -r))
    out = mlp(x, logits).float()
    assert bool(((out - expected).abs() <= 2 ** -7 * expected.abs() + 1e-6 * expected.abs().max()).all())


@pytest.mark.parametrize("T", [1, 16, 200])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_expert_mlp_takes_logits_with_overlapping_rows(T, dtype):
    """Logits whose rows share memory: one row for all tokens (stride 0), and rows that start one expert apart."""
    mlp = _small_expert_mlp(1)[2]
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, mlp.K, generator=g).to(torch.bfloat16).to(DEV)
    flat = torch.randperm(T + mlp.E, generator=g).to(dtype).to(DEV)
    for logits in (flat[:mlp.E].expand(T, mlp.E), flat.as_strided((T, mlp.E), (1, 1)), flat[:mlp.E].flip(0).expand(T, mlp.E)):
        assert torch.equal(mlp(x, logits), mlp(x, logits.contiguous()))


@pytest.mark.parametrize("num_rows", [1, 200, 256, 300, 511, 600])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_routed_gemm_with_a_row_count_inside_a_block(num_rows, out_dtype):
    """num_rows that is not whole 256-row blocks (or lies past the buffers): the rows below it are computed, the blocks at or past it are
    left alone."""
    from test_gpu_parity import check, random_problem
    R, N, K = 512, 320, 256
    a, a_s, _, _ = random_problem(R, 1, K, seed=9)
    weights = [random_problem(1, N, K, seed=10 + e)[2:] for e in range(2)]
    experts = ExpertWeights([b.to(DEV) for b, _ in weights], [s.to(DEV) for _, s in weights])
    c = torch.full((R, N), -1.0, dtype=out_dtype, device=DEV)
    moe.moe_scaled_gemm(a.to(DEV), a_s.to(DEV), experts, torch.tensor([1, 0], dtype=torch.int32, device=DEV),
                        torch.tensor([num_rows], dtype=torch.int32, device=DEV), c)
    for block, (b, b_s) in ((0, weights[1]), (1, weights[0])):
        lo, hi = 256 * block, min(256 * (block + 1), num_rows)
        if lo < hi:
            check(c[lo:hi], a[lo:hi], a_s[lo:hi], b, b_s)
        else:
            assert bool((c[lo:] == -1.0).all())


@pytest.mark.parametrize("T,E,k", [(127, 32, 32), (128, 9, 3), (129, 8, 8), (257, 32, 5), (8192, 8, 1), (8193, 17, 2), (20001, 32, 4)])
def test_expert_mlp_routes_blocks_of_tokens(T, E, k):
    """The routing of the single call at its edges: one launch and two, the last block of tokens partly filled, blocks of more than 128
    tokens, every expert chosen, experts without tokens. Against the same steps one by one, whose rows are sorted by
    moe_align_block_size; the outputs differ by the summation order of the last GEMM at most (one bf16 ulp of a term)."""
    K = inter = 128
    _, _, mlp = _small_expert_mlp(T + E, E=E, K=K, inter=inter, N=32, k=k)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    logits = torch.randn(T, E, generator=g)
    if E > k + 2:
        logits[:, 1] = -50.0  # an expert without tokens
    logits = logits.to(DEV)
    assert mlp._takes_fused(x, logits)
    y, ref = mlp(x, logits), mlp._forward_steps(x, logits)
    assert y.shape == ref.shape and bool(torch.isfinite(y.float()).all())
    assert float((y.float() - ref.float()).abs().max()) <= 2 ** -7 * float(ref.float().abs().max())
    ops.check_device_status()
