"""GPU parity: the CUDA kernels, called through the C ABI and through the template API, against the
CPU oracle and the golden vectors made from the reference. Mirrors the reference's own MXFP4 tests
(tests/kernel/wave_gemm_mxfp_test.py, tests/kernel/wave_gemm_test.py:3640-3690).

Tolerances (stated by the task this library serves):
  * dequantised operands and repacked scales: bit-exact;
  * f32 output: |c - ref| <= 1e-5 * |ref| + 1e-5 * sqrt(K) * max|row of dequant(a)| * max|row of dequant(b)|;
  * bf16 output: within 1 bf16 ulp of the f32 reference rounded to bf16.
"""

import ctypes
import functools

import numpy as np
import pytest
import torch

import wave_b200 as wb
from conftest import GOLDEN
from oracle import mxfp4_oracle as orc
from wave_b200 import _lib, ops

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def check_f32(c, a, a_s, b, b_s, ref=None):
    K = a.shape[1] * 2
    if ref is None:
        ref = orc.scaled_gemm(a, a_s, b, b_s)
    tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s), orc.dequant_mxfp4(b, b_s), ref, K)
    err = (c.float().cpu() - ref).abs()
    bad = ~(err <= tol)
    assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} outside tolerance, max err {float(err.max())}"


def check_bf16(c, ref):
    d = orc.bf16_ulp_distance(c, ref)
    assert int(d.max()) <= 1, f"{int((d > 1).sum())} of {d.numel()} differ by more than 1 bf16 ulp (max {int(d.max())})"


def check(c, a, a_s, b, b_s, ref=None):
    if ref is None:
        ref = orc.scaled_gemm(a, a_s, b, b_s)
    if c.dtype == torch.float32:
        check_f32(c, a, a_s, b, b_s, ref)
    else:
        check_bf16(c, ref)
    ops.check_device_status()


def random_problem(M, N, K, seed, lo=124, hi=131):
    g = torch.Generator().manual_seed(seed)
    a = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, generator=g)
    b = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g)
    a_s = torch.randint(lo, hi, (M, K // 32), dtype=torch.uint8, generator=g)
    b_s = torch.randint(lo, hi, (N, K // 32), dtype=torch.uint8, generator=g)
    return a, a_s, b, b_s


def quantized_problem(M, N, K, seed_a, seed_b, std_b=1.0):
    a, a_s = orc.quantize_mxfp4(torch.randn(M, K, generator=torch.Generator().manual_seed(seed_a)))
    b, b_s = orc.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(seed_b)) * std_b)
    return a, a_s, b, b_s


def run(a, a_s, b, b_s, out_dtype=torch.float32, path=_lib.PATH_AUTO, fill=float("nan")):
    kernel, options = wb.get_tagged_mxfp4_gemm((a.shape[0], b.shape[0], a.shape[1] * 2),
                                               output_dtype=wb.TORCH_DTYPE_TO_WAVE[out_dtype])
    options.kernel_path = path
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    c = torch.full((a.shape[0], b.shape[0]), fill, dtype=out_dtype, device=DEV)  # kernel must overwrite all of c
    gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
    return c


# ---------------------------------------------------------------------------------------------
# scale repack and dequantisation: bit-exact
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("rows,K", [(128, 256), (1024, 1024), (100, 96), (300, 8192), (16, 8192), (257, 1184),
                                    (1, 32), (4096, 16384)])
def test_repack_scales_bit_exact(rows, K):
    s = torch.randint(0, 256, (rows, K // 32), dtype=torch.uint8)
    got = ops.repack_scales(s.to(DEV))
    assert torch.equal(got.data.cpu(), orc.pack_scales(s))
    assert got.data.numel() == ops.packed_scale_bytes(rows, K)


def test_repack_scales_strided_source():
    s = torch.randint(0, 256, (70, 40), dtype=torch.uint8)
    view = s.to(DEV)[:, 3:19]  # row stride 40, 16 K-blocks, misaligned start
    got = ops.repack_scales(view)
    assert torch.equal(got.data.cpu(), orc.pack_scales(s[:, 3:19].contiguous()))


@pytest.mark.parametrize("rows,K", [(64, 256), (33, 96), (1000, 4096)])
def test_dequant_bit_exact_all_codes(rows, K):
    q = torch.randint(0, 256, (rows, K // 2), dtype=torch.uint8)
    s = torch.randint(0, 256, (rows, K // 32), dtype=torch.uint8)  # includes 0, 254 and the NaN code 255
    got = wb.mxfp4_dequant(q.to(DEV), s.to(DEV)).cpu()
    exp = orc.dequant_mxfp4(q, s)
    same = (got.view(torch.int32) == exp.view(torch.int32)) | (got.isnan() & exp.isnan())
    assert bool(same.all()), f"{int((~same).sum())} mismatches"


def test_dequant_golden_edges():
    g = np.load(GOLDEN / "gemm_wide_scales_48x80x256.npz")
    a = torch.from_numpy(g["a"])
    for scale_key, deq_key in (("a_scale", "a_deq"), ("edge_scale", "edge_deq")):
        got = wb.mxfp4_dequant(a.to(DEV), torch.from_numpy(g[scale_key]).to(DEV)).cpu().numpy()
        exp = g[deq_key]
        assert bool(((got.view(np.int32) == exp.view(np.int32)) | (np.isnan(got) & np.isnan(exp))).all())


# ---------------------------------------------------------------------------------------------
# golden GEMM vectors from the reference
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_golden_seed5_small(out_dtype):
    g = np.load(GOLDEN / "gemm_seed5_64x96x128.npz")
    x, w, xs, ws = (torch.from_numpy(g[k]) for k in ("x", "w", "x_scales", "w_scales"))
    c = run(x, xs, w.T.contiguous(), ws, out_dtype)
    check(c, x, xs, w.T.contiguous(), ws, ref=torch.from_numpy(g["out"]))


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_golden_wide_scales(out_dtype):
    g = np.load(GOLDEN / "gemm_wide_scales_48x80x256.npz")
    a, b, a_s, b_s = (torch.from_numpy(g[k]) for k in ("a", "b", "a_scale", "b_scale"))
    c = run(a, a_s, b, b_s, out_dtype)
    check(c, a, a_s, b, b_s, ref=torch.from_numpy(g["out"]))


def test_reference_test_shape_1024_seed5_f32():
    """testScaledGemmMXFP4 (wave_gemm_mxfp_test.py:94-201) at (1024, 1024, 1024), written as the reference writes it."""
    shape = (1024, 1024, 1024)
    kernel, hyper = wb.get_scaled_gemm_kernel(shape, wb.ScaledMMAType.F32_16x16x128_F8F6F4)
    options = wb.WaveCompileOptions(subs=hyper, canonicalize=True, schedule=wb.SchedulingType.NONE)
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    x, w, x_scales, w_scales = wb.generate_gemm_afp4wfp4_inputs(shape, device=torch.device("cpu"))
    ox, ow, oxs, ows = orc.generate_gemm_afp4wfp4_inputs(shape)
    assert torch.equal(x, ox) and torch.equal(w, ow) and torch.equal(x_scales, oxs) and torch.equal(w_scales, ows)
    out = torch.zeros(x.shape[0], w.shape[1], dtype=torch.float32, device=DEV)
    w_t = w.T.contiguous()
    gemm(x.to(DEV), x_scales.to(DEV), w_t.to(DEV), w_scales.to(DEV), out)
    torch_out = orc.torch_scaled_gemm_mxfp4(x, w, x_scales, w_scales)
    torch.testing.assert_close(torch_out, out.cpu(), check_dtype=False)  # the reference's own (default) tolerance
    check(out, x, x_scales, w_t, w_scales, ref=torch_out)
    g = np.load(GOLDEN / "gemm_seed5_1024_sample.npz")
    torch.testing.assert_close(out.cpu()[::64, ::64], torch.from_numpy(g["out_sample"]), rtol=1e-5, atol=1e-3)


def test_config1_1024_cubed_wide_scales_f32():
    """Scales uniform in [124, 130], codes uniform over all 16 values, f32 output."""
    x, w, xs, ws = orc.generate_gemm_afp4wfp4_inputs((1024, 1024, 1024), scale_lo=124, scale_hi=131)
    w_t = w.T.contiguous()
    check(run(x, xs, w_t, ws, torch.float32), x, xs, w_t, ws)


# ---------------------------------------------------------------------------------------------
# every kernel path, ragged and aligned shapes, both output types
# ---------------------------------------------------------------------------------------------
TILE_PATHS = [_lib.PATH_TILE_1CTA, _lib.PATH_TILE_1CTA | _lib.TILE_N128, _lib.PATH_TILE_2CTA,
              _lib.PATH_TILE_2CTA | _lib.TILE_N128, _lib.PATH_TILE_1CTA | _lib.TILE_N192,
              _lib.PATH_TILE_2CTA | _lib.TILE_N192]


@pytest.mark.parametrize("flags", TILE_PATHS)
@pytest.mark.parametrize("shape", [(128, 128, 256), (256, 512, 1024), (1000, 1100, 992), (130, 260, 32),
                                   (1024, 1600, 2048), (512, 1920, 1024), (3, 5, 64)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_tile_paths(flags, shape, out_dtype):
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K)
    ad, asd, bd, bsd = a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV)
    c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, ops.repack_scales(asd), bd, ops.repack_scales(bsd), c, flags)
    check(c, a, a_s, b, b_s)


@pytest.mark.parametrize("M", [1, 4, 16, 17, 64, 100, 128])
@pytest.mark.parametrize("N,K", [(1024, 2048), (1000, 992), (4096, 512)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_skinny_path(M, N, K, out_dtype):
    a, a_s, b, b_s = random_problem(M, N, K, seed=7 * M + N)
    c = run(a, a_s, b, b_s, out_dtype, path=_lib.PATH_SKINNY)
    check(c, a, a_s, b, b_s)
    # the same launch again gives the same bits (fixed-order reduction; counters left clean)
    c2 = run(a, a_s, b, b_s, out_dtype, path=_lib.PATH_SKINNY)
    assert torch.equal(c.view(torch.int16 if out_dtype == torch.bfloat16 else torch.int32),
                       c2.view(torch.int16 if out_dtype == torch.bfloat16 else torch.int32))


@pytest.mark.parametrize("shape", [(1024, 2304, 512), (640, 5120, 256)])
def test_raster_group_changes_the_tile_order_not_the_result(shape):
    """WB200_GROUP_N (the templates' reorder_workgroups / group_size_n): every group size gives the bits of the default."""
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=4242)
    ad, bd = a.to(DEV), b.to(DEV)
    asp, bsp = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    for path in (_lib.PATH_TILE_1CTA, _lib.PATH_TILE_2CTA):
        base = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.scaled_gemm_packed(ad, asp, bd, bsp, base, path)
        check(base, a, a_s, b, b_s)
        for group in (_lib.GROUP_N(1), _lib.GROUP_N(3), _lib.GROUP_N(32), _lib.GROUP_N(254), _lib.GROUP_N_ALL):
            c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
            ops.scaled_gemm_packed(ad, asp, bd, bsp, c, path | group)
            assert torch.equal(c.view(torch.int16), base.view(torch.int16))


def test_template_group_size_reaches_the_kernel():
    """get_tagged_mxfp4_gemm(group_size_n=..., reorder_workgroups=...) compiles to the matching raster flags and
    still matches the oracle."""
    M, N, K = 512, 2048, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=77)
    for kwargs, want in ((dict(group_size_n=4), _lib.GROUP_N(4)), (dict(group_size_n=8, block_shape=(256, 128, 256)), _lib.GROUP_N(4)),
                         (dict(reorder_workgroups=False), _lib.GROUP_N_ALL), (dict(), 0)):
        tpl, options = wb.templates.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16, **kwargs)
        gemm = wb.wave_compile(options, tpl)
        assert gemm._raster_flags() == want
        c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
        check(c, a, a_s, b, b_s)


def test_many_tiles_per_cta_and_accumulator_reuse():
    """More tiles than SMs on every path, so each CTA runs several tiles through both accumulators."""
    M, N, K = 2048, 6144, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=99)
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    ad, bd = a.to(DEV), b.to(DEV)
    asp, bsp = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    for flags in TILE_PATHS:
        for out_dtype in (torch.bfloat16, torch.float32):
            c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
            ops.scaled_gemm_packed(ad, asp, bd, bsp, c, flags)
            check(c, a, a_s, b, b_s, ref=ref)


def test_output_column_block_with_row_pitch():
    """c may be a column block of a wider matrix (what the N-sharded launcher writes into)."""
    M, N, K = 256, 384, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=5)
    wide = torch.full((M, 1024), -7.0, dtype=torch.bfloat16, device=DEV)
    ad, bd = a.to(DEV), b.to(DEV)
    ops.scaled_gemm_packed(ad, ops.repack_scales(a_s.to(DEV)), bd, ops.repack_scales(b_s.to(DEV)), wide[:, 256:640])
    check_bf16(wide[:, 256:640].contiguous(), orc.scaled_gemm(a, a_s, b, b_s))
    assert bool((wide[:, :256] == -7.0).all()) and bool((wide[:, 640:] == -7.0).all())


def test_unaligned_output_falls_back_to_scalar_stores():
    M, N, K = 130, 70, 256
    a, a_s, b, b_s = random_problem(M, N, K, seed=11)
    wide = torch.zeros(M, 75, dtype=torch.float32, device=DEV)  # row pitch 300 bytes: not a multiple of 16
    ops.scaled_gemm_packed(a.to(DEV), ops.repack_scales(a_s.to(DEV)), b.to(DEV), ops.repack_scales(b_s.to(DEV)),
                           wide[:, 3:73], _lib.PATH_TILE_1CTA)
    check_f32(wide[:, 3:73].contiguous(), a, a_s, b, b_s)


# ---------------------------------------------------------------------------------------------
# reference API variants
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("shape,num_splits", [((256, 256, 256), 2), ((256, 256, 512), 4), ((256, 256, 1024), 4),
                                              ((512, 512, 1024), 4)])
@pytest.mark.parametrize("output_type", [torch.float32, torch.bfloat16])
def test_splitk_adds_into_c(shape, num_splits, output_type):
    """testSplitKMxfp4Gemm (wave_gemm_test.py:3640-3690): zero-initialised c, result added in."""
    kernel, options = wb.get_tagged_splitk_mxfp4_gemm(shape, num_splits=num_splits, block_shape=(128, 128, 128),
                                                      output_type=wb.TORCH_DTYPE_TO_WAVE[output_type])
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel, wb.get_mxfp4_dbuf_schedule(True, 1))
    x, w, xs, ws = orc.generate_gemm_afp4wfp4_inputs(shape)
    ref = orc.torch_scaled_gemm_mxfp4(x, w, xs, ws)
    w_t = w.T.contiguous()
    c = torch.zeros(shape[0], shape[1], dtype=output_type, device=DEV)
    gemm(x.to(DEV), xs.to(DEV), w_t.to(DEV), ws.to(DEV), c)
    check(c, x, xs, w_t, ws, ref=ref)  # far inside the reference's rtol 1e-3 / atol 1e-2 (f32) and atol 4.0 (bf16)
    if output_type == torch.float32:
        gemm(x.to(DEV), xs.to(DEV), w_t.to(DEV), ws.to(DEV), c)  # second call accumulates: c == 2 * ref
        torch.testing.assert_close(c.cpu(), 2 * ref, rtol=1e-5, atol=1e-2)


def test_splitk_skinny_accumulates():
    M, N, K = 16, 512, 2048
    a, a_s, b, b_s = random_problem(M, N, K, seed=21)
    kernel, options = wb.get_tagged_splitk_mxfp4_gemm((M, N, K), num_splits=2)
    gemm = wb.wave_compile(options, kernel)
    c = torch.ones(M, N, dtype=torch.float32, device=DEV)
    gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
    ref = orc.scaled_gemm(a, a_s, b, b_s) + 1.0
    check_f32(c, a, a_s, b, b_s, ref=ref)


def test_batched_activations_shared_weights():
    """testScaledBatchedGemmMXFP4 (wave_gemm_mxfp_test.py:205-339): a is [B, M, K/2], b is shared."""
    B, M, N, K = 4, 96, 256, 512
    a, a_s, b, b_s = random_problem(B * M, N, K, seed=31)
    kernel, options = wb.get_tagged_mxfp4_gemm((B * M, N, K))
    options.dynamic_symbols = ["M", "N", "K"]
    gemm = wb.wave_compile(options, kernel)
    c = torch.empty(B, M, N, dtype=torch.float32, device=DEV)
    gemm(a.view(B, M, -1).to(DEV), a_s.view(B, M, -1).to(DEV), b.to(DEV), b_s.to(DEV), c)
    check_f32(c.view(B * M, N), a, a_s, b, b_s)


def test_preshuffled_scale_templates():
    shape = (256, 384, 1024)
    a, a_s, b, b_s = random_problem(*shape, seed=41)
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    for make in (wb.get_tagged_mxfp4_gemm_preshuffle_scales, wb.get_tagged_mxfp4_gemm_preshuffle_scales_and_B,
                 wb.get_tagged_mxfp4_gemm_preshuffle_b, wb.get_tagged_mxfp4_gemm_preshuffle_b_wide_store):
        kernel, options = make(shape, output_dtype=wb.bf16)
        gemm = wb.wave_compile(options, kernel)
        c = torch.empty(shape[0], shape[1], dtype=torch.bfloat16, device=DEV)
        gemm(a.to(DEV), wb.e8m0_shuffle(a_s.to(DEV)), wb.b_preshuffle(b.to(DEV)), wb.e8m0_shuffle(b_s.to(DEV)), c)
        check_bf16(c, ref)
        with pytest.raises(ValueError, match="pre-shuffled"):
            gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)


def test_call_time_errors():
    kernel, options = wb.get_tagged_mxfp4_gemm((64, 64, 64))
    gemm = wb.wave_compile(options, kernel)
    a = torch.zeros(64, 32, dtype=torch.uint8, device=DEV)
    s = torch.zeros(64, 2, dtype=torch.uint8, device=DEV)
    with pytest.raises(ValueError, match="writes f32"):
        gemm(a, s, a, s, torch.zeros(64, 64, dtype=torch.bfloat16, device=DEV))
    with pytest.raises(ValueError, match="was built for"):
        gemm(a[:32], s[:32], a, s, torch.zeros(32, 64, device=DEV))
    with pytest.raises(ValueError, match="a_scale must be"):
        gemm(a, s[:, :1], a, s, torch.zeros(64, 64, device=DEV))
    with pytest.raises(ValueError, match="uint8 or int8"):
        gemm(a.float(), s, a, s, torch.zeros(64, 64, device=DEV))
    with pytest.raises(ValueError, match="workspace"):
        _lib.check(_lib.load().wb200_mxfp4_gemm(16, 64, 64, a.data_ptr(), a.data_ptr(), a.data_ptr(), a.data_ptr(),
                                                a.data_ptr(), 0, 64, None, 0, _lib.PATH_SKINNY, None))
    assert ctypes.c_int(_lib.load().wb200_version()).value >= 1000


def test_noncontiguous_inputs_are_copied():
    M, N, K = 64, 128, 256
    a, a_s, b, b_s = random_problem(M, N, K, seed=51)
    a_wide = torch.zeros(M, K, dtype=torch.uint8, device=DEV)
    a_wide[:, ::2] = a.to(DEV)
    c = torch.empty(M, N, device=DEV)
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K))
    wb.wave_compile(options, kernel)(a_wide[:, ::2], a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
    check_f32(c, a, a_s, b, b_s)


# ---------------------------------------------------------------------------------------------
# full-size configurations: sampled oracle rows plus size-independent properties
# ---------------------------------------------------------------------------------------------
def test_config2_8192_cubed_bf16_whole_matrix_and_scaling_property():
    """M = N = K = 8192, operands quantised from N(0, 1), bf16 output. The whole output is compared with the
    oracle, 512 rows of A at a time (the reference's tests compare whole outputs too,
    tests/kernel/wave_gemm_mxfp_test.py:184-201), and through an exact property: raising every A scale by one
    doubles C bit for bit (power-of-two scaling is exact)."""
    M = N = K = 8192
    a, a_s, b, b_s = quantized_problem(M, N, K, 1002, 2002)
    ad, asd, bd, bsd = a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV)
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)
    c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    gemm(ad, asd, bd, bsd, c)
    c_host = c.cpu()
    b_deq = orc.dequant_mxfp4(b, b_s)  # once: 256 MB of f32
    for r0 in range(0, M, 512):
        ref = orc.dequant_mxfp4(a[r0:r0 + 512], a_s[r0:r0 + 512]) @ b_deq.T
        check_bf16(c_host[r0:r0 + 512], ref)
    del b_deq
    c2 = torch.empty_like(c)
    gemm(ad, asd + 1, bd, bsd, c2)
    assert torch.equal((c.float() * 2).to(torch.bfloat16), c2)
    ops.check_device_status()


@functools.lru_cache(maxsize=1)
def _config3_operands():
    N, K = 28672, 8192
    a, a_s = orc.quantize_mxfp4(torch.randn(128, K, generator=torch.Generator().manual_seed(1003)))
    b, b_s = orc.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(2003)) * 0.02)
    return a, a_s, b, b_s


@pytest.mark.parametrize("M", [1, 4, 16, 64, 128])
def test_config3_decode_shapes_bf16(M):
    """N = 28672, K = 8192, weights from N(0, 0.02), activations from N(0, 1); column blocks of the
    oracle are checked (the full dequantised weight matrix would be 0.9 GB)."""
    N = 28672
    a, a_s, b, b_s = _config3_operands()
    a, a_s = a[:M].contiguous(), a_s[:M].contiguous()
    c = run(a, a_s, b, b_s, torch.bfloat16)
    # every column block at M = 16 (the shape the bandwidth target is quoted on), three of them otherwise
    blocks = range(0, N, 2048) if M == 16 else (0, 12288, N - 2048)
    for n0 in blocks:
        ref = orc.scaled_gemm(a, a_s, b[n0:n0 + 2048], b_s[n0:n0 + 2048])
        check_bf16(c[:, n0:n0 + 2048].contiguous(), ref)
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K,out_dtype,accumulate", [
    (16, 28672, 2048, torch.bfloat16, False),   # one static round, 76 dealt tiles in main / closer parts
    (16, 28672 + 72, 1024, torch.float32, False),  # ragged last tile among the dealt ones
    (100, 19200, 1536, torch.bfloat16, False),  # 150 tiles: 2 dealt tiles only
    (4, 18944, 512, torch.float32, True),       # a whole number of rounds; accumulate into c
    (16, 38000, 256, torch.bfloat16, False),    # one K block per tile: nothing to cut
])
def test_skinny_path_with_dealt_parts(M, N, K, out_dtype, accumulate):
    """Shapes with at least as many N tiles as SMs: the kernel that deals whole N tiles from an atomic counter.
    Checked against the oracle; and because which CTA computes which tile varies from run to run while each
    tile's sum over K does not, repeated launches must give the same bits."""
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K, lo=124, hi=128)
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    ad, bd = a.to(DEV), b.to(DEV)
    a_sf, b_sf = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    flags = _lib.PATH_SKINNY | (_lib.ACCUMULATE if accumulate else 0)
    outs = []
    for _ in range(4):
        c = torch.full((M, N), 1.0 if accumulate else float("nan"), dtype=out_dtype, device=DEV)
        ops.scaled_gemm_packed(ad, a_sf, bd, b_sf, c, flags)
        outs.append(c)
    check(outs[0], a, a_s, b, b_s, ref + 1.0 if accumulate else ref)
    bits = torch.int16 if out_dtype == torch.bfloat16 else torch.int32
    for c in outs[1:]:
        assert torch.equal(outs[0].view(bits), c.view(bits))


@pytest.mark.parametrize("rows,K,tile_rows", [(300, 768, 104), (28672 // 8, 512, 104), (97, 96, 96), (1000, 256, 8), (256, 1024, 128),
                                              (224, 256, 224), (1000, 288, 224), (8192, 512, 224)])
def test_tiled_weight_scale_packing_is_bit_exact(rows, K, tile_rows):
    s = torch.randint(0, 255, (rows, K // 32), dtype=torch.uint8, generator=torch.Generator().manual_seed(rows + tile_rows))
    packed = ops.repack_scales(s.to(DEV), tile_rows=tile_rows)
    assert packed.tile_rows == tile_rows
    assert torch.equal(packed.data.cpu(), orc.pack_scales_tiled(s, tile_rows))


@pytest.mark.parametrize("M", [1, 16, 40, 128])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_decode_kernel_with_weight_scales_packed_per_balanced_tile(M, out_dtype):
    """N = 28672 (the decode configuration's N): the balanced tile height is below 128 on any part whose SM count
    does not divide 224; the GEMM on scales packed for it matches the oracle, and gives the bits of the usual packing
    (every output column's sum over K is made in the same order either way)."""
    N, K = 28672, 256
    h = ops.decode_tile_rows(N)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert h % 8 == 0 and 8 <= h <= 128
    if 224 % sms:
        assert h < 128 and -(-N // h) <= -(-224 // sms) * sms  # every SM gets at most `rounds` tiles
    a, a_s, b, b_s = random_problem(M, N, K, seed=500 + M)
    ad, bd = a.to(DEV), b.to(DEV)
    a_sf = ops.repack_scales(a_s.to(DEV))
    usual, tiled = ops.repack_scales(b_s.to(DEV)), ops.repack_scales(b_s.to(DEV), tile_rows=h)
    c0 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    c1 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, usual, c0, _lib.PATH_SKINNY)
    ops.scaled_gemm_packed(ad, a_sf, bd, tiled, c1, _lib.PATH_SKINNY)
    check(c1, a, a_s, b, b_s)
    bits = torch.int16 if out_dtype == torch.bfloat16 else torch.int32
    assert torch.equal(c0.view(bits), c1.view(bits))
    # accumulate form and a ragged N on the same packing rule
    N2 = N - 200
    h2 = ops.decode_tile_rows(N2)
    t2 = ops.repack_scales(b_s[:N2].to(DEV), tile_rows=h2)
    c2 = torch.ones(M, N2, dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd[:N2].contiguous(), t2, c2, _lib.PATH_SKINNY | _lib.ACCUMULATE)
    check(c2, a, a_s, b[:N2], b_s[:N2], orc.scaled_gemm(a, a_s, b[:N2], b_s[:N2]) + 1.0)


@pytest.mark.parametrize("shape", [(256, 224, 256), (300, 1000, 288), (1024, 2304, 1024), (2048, 4096, 512)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_224_wide_tiles_on_weight_scales_packed_for_them(shape, out_dtype):
    """CTA-pair tiles of 224 columns: two accumulators side by side in tensor memory (no hand-over between tiles), read
    from weight scales packed two atom rows per 224-row tile. Same bits as the 256-wide kernel (each output's sum over
    K is made in the same order)."""
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N)
    ad, bd, a_sf = a.to(DEV), b.to(DEV), ops.repack_scales(a_s.to(DEV))
    c224 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, ops.repack_scales(b_s.to(DEV), tile_rows=224), c224)
    check(c224, a, a_s, b, b_s)
    c256 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, ops.repack_scales(b_s.to(DEV)), c256, _lib.PATH_TILE_2CTA)
    bits = torch.int16 if out_dtype == torch.bfloat16 else torch.int32
    assert torch.equal(c224.view(bits), c256.view(bits))
    with pytest.raises(Exception):  # forcing another width on scales packed for 224 is refused
        ops.scaled_gemm_packed(ad, a_sf, bd, ops.repack_scales(b_s.to(DEV), tile_rows=224), c224, _lib.PATH_TILE_2CTA | _lib.TILE_N128)
    ops.check_device_status()


@pytest.mark.parametrize("shape", [(256, 448, 10240), (300, 1000, 16000), (129, 224, 12288), (700, 900, 10272)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_224_wide_tiles_with_few_tiles_and_a_long_k(shape, out_dtype):
    """The sizes at which the usual packing of the weight scales goes to the cluster split-K kernel, whose 128-wide tiles cannot
    read a packing per 224 rows: the call stays on the 224-wide tile kernel. One N tile, several, and a ragged last one."""
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N)
    ad, bd, a_sf = a.to(DEV), b.to(DEV), ops.repack_scales(a_s.to(DEV))
    c224 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, ops.repack_scales(b_s.to(DEV), tile_rows=224), c224)
    check(c224, a, a_s, b, b_s)
    c256 = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, ops.repack_scales(b_s.to(DEV)), c256, _lib.PATH_TILE_2CTA)
    bits = torch.int16 if out_dtype == torch.bfloat16 else torch.int32
    assert torch.equal(c224.view(bits), c256.view(bits))


def test_tiled_weight_scales_are_refused_where_no_kernel_reads_them():
    N, K = 28672, 256
    h = ops.decode_tile_rows(N)
    if h == 128:
        pytest.skip("this part's SM count divides the tile count: no tiled packing")
    a, a_s, b, b_s = random_problem(256, N, K, seed=9)
    tiled = ops.repack_scales(b_s.to(DEV), tile_rows=h)
    c = torch.empty(256, N, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(ValueError):  # M > 128: the tile kernels read 128-row blocks
        ops.scaled_gemm_packed(a.to(DEV), ops.repack_scales(a_s.to(DEV)), b.to(DEV), tiled, c)
    lib = _lib.load()
    small = ops.repack_scales(b_s[:1024].to(DEV), tile_rows=h)  # fewer tiles than SMs
    c16 = torch.empty(16, 1024, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(Exception) as err:
        ops.scaled_gemm_packed(a[:16].to(DEV), ops.repack_scales(a_s[:16].to(DEV)), b[:1024].to(DEV), small, c16, _lib.PATH_SKINNY)
    assert "wb200_repack_scales" in str(err.value)
    assert lib.wb200_packed_scale_bytes_tiled(100, 256, 100) == 0  # not a multiple of 8
    ops.check_device_status()


def test_template_call_packs_weight_scales_for_the_decode_kernel():
    """The reference-facing call at M <= 128 uses the balanced packing by itself and keeps the usual one for M > 128
    of the same weight; both match the oracle."""
    N, K = 28672, 256
    a, a_s, b, b_s = random_problem(256, N, K, seed=77)
    tpl, options = wb.templates.get_tagged_mxfp4_gemm((16, N, K), output_dtype=wb.bf16)
    tpl.shape = None  # dynamic M
    gemm = wb.wave_compile(options, tpl)
    bd, bsd = b.to(DEV), b_s.to(DEV)
    for M in (16, 256, 16):
        c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        gemm(a[:M].to(DEV), a_s[:M].to(DEV), bd, bsd, c)
        check(c, a[:M], a_s[:M], b, b_s)
    h = ops.decode_tile_rows(N)
    heights = sorted({k[-1] for k in gemm._weight_scales._entries})
    assert heights == sorted({h, 128})


def test_two_streams_run_skinny_gemms_at_the_same_time():
    """Two decode-shaped GEMMs launched on two streams with nothing ordering them: each call gets its own
    workspace (counters and partial tiles belong to one running GEMM), so both match the oracle however the
    GPU interleaves them."""
    M, N, K = 16, 20480, 1024
    probs = [random_problem(M, N, K, seed=s, lo=124, hi=128) for s in (11, 12)]
    refs = [orc.scaled_gemm(*p) for p in probs]
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)  # ONE kernel object, used from both streams
    dev = [[t.to(DEV) for t in p] for p in probs]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in probs]
    streams = [torch.cuda.Stream(DEV) for _ in probs]
    torch.cuda.synchronize()
    for rep in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                gemm(*dev[i], outs[i])
    torch.cuda.synchronize()
    for i in range(2):
        check_bf16(outs[i], refs[i])
    ops.check_device_status()


def test_workspace_of_a_captured_call_outlives_a_larger_call(monkeypatch):
    """The graph of a decode GEMM writes its counters and partial tiles where the workspace was at the capture. Blocks of that size
    that are allocated after a larger call has made a new workspace are not written by a replay."""
    monkeypatch.setattr(ops, "_pool", ops.WorkspacePool())
    N, K = 4096, 16384  # at 16 rows the K-split kernel, which uses the workspace
    a, a_s, b, b_s = random_problem(128, N, K, seed=78)
    a_sf, b_sf = [ops.repack_scales(a_s[:m].to(DEV)) for m in (16, 128)], ops.repack_scales(b_s.to(DEV))
    ad, bd = a.to(DEV), b.to(DEV)
    c = torch.empty(16, N, dtype=torch.bfloat16, device=DEV)
    stream, graph = torch.cuda.Stream(DEV), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        ops.scaled_gemm_packed(ad[:16], a_sf[0], bd, b_sf, c, _lib.PATH_SKINNY)
    torch.cuda.synchronize()
    ref = c.clone()
    with torch.cuda.graph(graph, stream=stream):
        ops.scaled_gemm_packed(ad[:16], a_sf[0], bd, b_sf, c, _lib.PATH_SKINNY)
    key = (0, stream.cuda_stream, "skinny")
    small = ops._pool._by_key[key].data_ptr(), ops._pool._by_key[key].numel()
    with torch.cuda.stream(stream):
        ops.scaled_gemm_packed(ad, a_sf[1], bd, b_sf, torch.empty(128, N, dtype=torch.bfloat16, device=DEV), _lib.PATH_SKINNY)
        assert ops._pool._by_key[key].numel() >= 2 * small[1]
        blocks = [torch.full((small[1],), 7, dtype=torch.uint8, device=DEV) for _ in range(4)]
    torch.cuda.synchronize()
    assert all(not (t.data_ptr() < small[0] + small[1] and small[0] < t.data_ptr() + t.numel()) for t in blocks)
    c.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c.view(torch.int16), ref.view(torch.int16)) and all(bool((t == 7).all()) for t in blocks)


@pytest.mark.parametrize("kind,M,N,K", [("fp4", 64, 28672, 1024), ("fp4", 256, 4096, 4096), ("fp4", 16, 1024, 12320), ("fp8", 16, 14336, 2048),
                                        ("mixed", 64, 28672, 2048), ("fp8", 300, 4096, 2048)])
def test_two_streams_pack_activation_scales_at_the_same_time(kind, M, N, K):
    """ONE kernel object called from two unordered streams at sizes whose activation scales are packed ahead of the GEMM (decode
    above 32 rows, tile and cluster kernels, rows of scales that are not whole 8-byte words, 8-bit operands): every stream
    packs into memory of its own. The scales of the two problems are powers of two apart, so that a block read from the
    other one shows. Reference: the same call alone, bit for bit."""
    g = torch.Generator().manual_seed(M + N)
    if kind == "fp4":
        kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    else:
        kernel, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4, "f8e4m3fn", wb.bf16,
                                                       weight_format="f4e2m1fn" if kind == "mixed" else None)
        options = wb.WaveCompileOptions(subs=subs)
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)

    def operand(rows, bits):
        t = torch.randint(0, 256, (rows, K * bits // 8), dtype=torch.uint8, generator=g)
        return (t if bits == 4 else (t & 0xBF).view(torch.float8_e4m3fn)).to(DEV)

    b = operand(N, 8 if kind == "fp8" else 4)
    b_s = torch.randint(124, 131, (N, K // 32), dtype=torch.uint8, generator=g).to(DEV)
    xs = [(operand(M, 4 if kind == "fp4" else 8), torch.randint(110 + 20 * i, 115 + 20 * i, (M, K // 32), dtype=torch.uint8, generator=g).to(DEV))
          for i in range(2)]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in xs]
    refs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in xs]
    for (a, a_s), c in zip(xs, refs):
        gemm(a, a_s, b, b_s, c)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream(DEV) for _ in xs]
    for rep in range(20):
        for st, (a, a_s), c in zip(streams, xs, outs):
            with torch.cuda.stream(st):
                gemm(a, a_s, b, b_s, c)
    torch.cuda.synchronize()
    for c, ref in zip(outs, refs):
        assert torch.equal(c.view(torch.int16), ref.view(torch.int16))
    ops.check_device_status()


def test_graphed_calls_of_one_object_have_scratch_of_their_own_and_allocate_none():
    """Two graphs over one kernel object, each warmed up on a stream of its own, and an eager call: three scratches, none of them made
    during a capture. Replays of both graphs and eager calls on three streams at once give the results of the calls alone."""
    from wave_b200.graphs import GraphedScaledGemm
    M, N, K = 64, 28672, 1024
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    a, _, b, b_s = (t.to(DEV) for t in random_problem(M, N, K, seed=3))
    scales = [torch.randint(110 + 8 * i, 115 + 8 * i, (M, K // 32), dtype=torch.uint8, device=DEV) for i in range(3)]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    refs = []
    for a_s in scales:
        gemm(a, a_s, b, b_s, outs[0])
        torch.cuda.synchronize()
        refs.append(outs[0].clone())
    graphs = [GraphedScaledGemm(gemm, a, scales[i], b, b_s, outs[i]) for i in range(2)]
    made = {key: [t.data_ptr() for t in bufs] for key, bufs in gemm._a_scale_buf.items()}
    plans = {p[3].data_ptr() for p in gemm._plans.values()}
    assert len(made) == 3 and plans == {v[0] for v in made.values()}  # (main stream and two warm-ups; the captures use those)
    streams = [torch.cuda.Stream(DEV) for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(20):
        for st, run in zip(streams, (graphs[0].replay, graphs[1].replay, lambda: gemm(a, scales[2], b, b_s, outs[2]))):
            with torch.cuda.stream(st):
                run()
    torch.cuda.synchronize()
    for c, ref in zip(outs, refs):
        assert torch.equal(c.view(torch.int16), ref.view(torch.int16))
    ops.check_device_status()


def test_scratch_of_a_captured_call_outlives_a_larger_call():
    """A graph holds the address of the scratch it packs into: a larger call on the same stream takes new memory and leaves the old
    one to the graph, whatever is allocated afterwards."""
    N, K = 4096, 2048
    kernel, options = wb.get_tagged_mxfp4_gemm((64, N, K), output_dtype=wb.bf16)
    options.dynamic_symbols = ["M"]
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    a, a_s, b, b_s = (t.to(DEV) for t in random_problem(512, N, K, seed=77))
    c = torch.empty(64, N, dtype=torch.bfloat16, device=DEV)
    stream, graph = torch.cuda.Stream(DEV), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        gemm(a[:64], a_s[:64], b, b_s, c)
    torch.cuda.synchronize()
    ref = c.clone()
    with torch.cuda.graph(graph, stream=stream):
        gemm(a[:64], a_s[:64], b, b_s, c)
    small = list(gemm._a_scale_buf.values())[0][-1]
    with torch.cuda.stream(stream):
        gemm(a, a_s, b, b_s, torch.empty(512, N, dtype=torch.bfloat16, device=DEV))
    torch.cuda.synchronize()
    assert list(gemm._a_scale_buf.values())[0][0] is small and list(gemm._a_scale_buf.values())[0][-1] is not small
    c.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c.view(torch.int16), ref.view(torch.int16))


# ---------------------------------------------------------------------------------------------
# grouped (MoE) GEMM
# ---------------------------------------------------------------------------------------------
def _moe_problem(E, N, K, tokens, seed):
    from wave_b200 import grouped
    g = torch.Generator().manual_seed(seed)
    x, x_s = orc.quantize_mxfp4(torch.randn(tokens, K, generator=g))
    weights = [orc.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(seed + 1 + e)) * 0.02)
               for e in range(E)]
    logits = torch.randn(tokens, E, generator=g)
    rows, offsets = grouped.route_top_k(logits, 2)
    return x, x_s, weights, rows, offsets


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_grouped_gemm_ragged_experts(out_dtype):
    """Top-2 routing over 5 experts gives ragged per-expert row counts (one expert is starved on purpose)."""
    from wave_b200 import grouped
    E, N, K, tokens = 5, 640, 1024, 300
    x, x_s, weights, rows, offsets = _moe_problem(E, N, K, tokens, seed=61)
    # starve the last expert: move its rows to expert 0 by re-routing (keeps the offsets consistent)
    assert offsets[-1] == 2 * tokens and len(offsets) == E + 1
    a, a_s = x[rows], x_s[rows]
    experts = grouped.ExpertWeights([w.to(DEV) for w, _ in weights], [s.to(DEV) for _, s in weights])
    c = torch.full((a.shape[0], N), float("nan"), dtype=out_dtype, device=DEV)
    grouped.grouped_scaled_gemm(a.to(DEV), a_s.to(DEV), experts, offsets, c)
    for e in range(E):
        r0, r1 = offsets[e], offsets[e + 1]
        if r1 == r0:
            continue
        w, s = weights[e]
        check(c[r0:r1].contiguous(), a[r0:r1], a_s[r0:r1], w, s)


def test_grouped_gemm_with_an_empty_expert():
    from wave_b200 import grouped
    E, N, K = 3, 256, 512
    g = torch.Generator().manual_seed(71)
    a = torch.randint(0, 256, (200, K // 2), dtype=torch.uint8, generator=g)
    a_s = torch.randint(124, 131, (200, K // 32), dtype=torch.uint8, generator=g)
    ws = [(torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g),
           torch.randint(124, 131, (N, K // 32), dtype=torch.uint8, generator=g)) for _ in range(E)]
    offsets = [0, 130, 130, 200]  # expert 1 gets no rows
    experts = grouped.ExpertWeights([w.to(DEV) for w, _ in ws], [s.to(DEV) for _, s in ws])
    c = torch.full((200, N), float("nan"), dtype=torch.float32, device=DEV)
    grouped.grouped_scaled_gemm(a.to(DEV), a_s.to(DEV), experts, offsets, c)
    for e in (0, 2):
        r0, r1 = offsets[e], offsets[e + 1]
        check_f32(c[r0:r1].contiguous(), a[r0:r1], a_s[r0:r1], ws[e][0], ws[e][1])
    with pytest.raises(ValueError):
        grouped.grouped_scaled_gemm(a.to(DEV), a_s.to(DEV), experts, [0, 100, 200], c)


def test_config4_moe_8_experts_bf16_sampled():
    """8 experts of [14336, 4096], 4096 tokens, top-2: every expert's block is checked on sampled rows and
    a column block of the oracle."""
    from wave_b200 import grouped
    E, N, K, tokens = 8, 14336, 4096, 4096
    x, x_s = orc.quantize_mxfp4(torch.randn(tokens, K, generator=torch.Generator().manual_seed(1004)))
    weights = [orc.quantize_mxfp4(torch.randn(N, K, generator=torch.Generator().manual_seed(2004 + e)) * 0.02)
               for e in range(E)]
    logits = torch.randn(tokens, E, generator=torch.Generator().manual_seed(3004))
    rows, offsets = grouped.route_top_k(logits, 2)
    assert offsets[-1] == 8192
    a, a_s = x[rows], x_s[rows]
    experts = grouped.ExpertWeights([w.to(DEV) for w, _ in weights], [s.to(DEV) for _, s in weights])
    c = torch.empty(a.shape[0], N, dtype=torch.bfloat16, device=DEV)
    grouped.grouped_scaled_gemm(a.to(DEV), a_s.to(DEV), experts, offsets, c)
    for e in range(E):
        r0, r1 = offsets[e], offsets[e + 1]
        sample = torch.arange(r0, r1, max(1, (r1 - r0) // 48))
        w, s = weights[e]
        n0 = (e * 1792) % (N - 2048)
        ref = orc.scaled_gemm(a[sample], a_s[sample], w[n0:n0 + 2048], s[n0:n0 + 2048])
        check_bf16(c[sample.to(DEV)][:, n0:n0 + 2048].contiguous(), ref)
        # the rows at both ends of the expert's block, against all columns of a narrow slice
        edge = torch.tensor([r0, r1 - 1])
        ref_e = orc.scaled_gemm(a[edge], a_s[edge], w[:512], s[:512])
        check_bf16(c[edge.to(DEV)][:, :512].contiguous(), ref_e)
    ops.check_device_status()


def test_grouped_repack_matches_per_group_repack():
    import ctypes
    lib = _lib.load()
    K = 1184  # 37 K-blocks: ragged along K too
    offsets = [0, 130, 130, 131, 400, 1000]
    s = torch.randint(0, 256, (offsets[-1], K // 32), dtype=torch.uint8)
    blocks = [0]
    for g in range(len(offsets) - 1):
        blocks.append(blocks[-1] + (offsets[g + 1] - offsets[g] + 127) // 128)
    per_block = ops.packed_scale_bytes(128, K)
    out = torch.zeros(blocks[-1] * per_block, dtype=torch.uint8, device=DEV)
    E = len(offsets) - 1
    sd = s.to(DEV)
    _lib.check(lib.wb200_repack_scales_grouped(sd.data_ptr(), sd.stride(0), E, (ctypes.c_int * (E + 1))(*offsets),
                                               (ctypes.c_int * (E + 1))(*blocks), K, out.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream))
    got = out.cpu()
    for g in range(E):
        r0, r1 = offsets[g], offsets[g + 1]
        if r1 > r0:
            exp = orc.pack_scales(s[r0:r1])
            assert torch.equal(got[blocks[g] * per_block: blocks[g] * per_block + exp.numel()], exp), g


# ---------------------------------------------------------------------------------------------
# activation quantiser and the linear module built on it
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,K", [(128, 256), (100, 96), (300, 8192), (1, 32), (257, 1184)])
def test_quantizer_bit_exact_against_oracle(rows, K, dtype):
    g = torch.Generator().manual_seed(rows + K)
    x = torch.randn(rows, K, generator=g) * torch.exp(torch.randn(rows, 1, generator=g) * 3)  # wide range of row scales
    x[0, :32] = 0.0                                                 # an all-zero block
    x[-1, :32] = 0.0
    x[-1, :8] = torch.tensor([6.0, 0.25, 0.75, 2.5, 5.0, -0.25, -1.25, 3.5]) * 4  # midpoints (ties) after scaling by 4
    x = x.to(dtype)
    q, s, packed = wb.quantize_mxfp4(x.to(DEV))
    eq, es = orc.quantize_mxfp4(x.float())
    assert torch.equal(s.cpu(), es)
    assert torch.equal(q.cpu(), eq)
    assert torch.equal(packed.data.cpu(), orc.pack_scales(es))


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 12])
@pytest.mark.parametrize("rows,K", [(1, 32), (130, 416)])
def test_quantizer_writes_scale_arrays_that_start_at_any_byte(rows, K, offset):
    """The C entry with both scale arrays `offset` bytes into a buffer: the oracle's bytes, padding included, and nothing beside them."""
    x = torch.randn(rows, K, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16)
    q_ref, s_ref = orc.quantize_mxfp4(x.float())
    packed_ref = orc.pack_scales(s_ref)
    xd, q = x.to(DEV), torch.empty(rows, K // 2, dtype=torch.uint8, device=DEV)
    rm = torch.full((s_ref.numel() + 32,), 0xEE, dtype=torch.uint8, device=DEV)
    pk = torch.full((packed_ref.numel() + 32,), 0xEE, dtype=torch.uint8, device=DEV)
    _lib.check(_lib.load().wb200_quantize_mxfp4(xd.data_ptr(), _lib.WB200_BF16, K, rows, K, q.data_ptr(), rm.data_ptr() + offset,
                                                pk.data_ptr() + offset, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(q.cpu(), q_ref)
    for buf, ref in ((rm.cpu(), s_ref.reshape(-1)), (pk.cpu(), packed_ref.reshape(-1))):
        assert torch.equal(buf[offset:offset + ref.numel()], ref)
        assert bool((buf[:offset] == 0xEE).all()) and bool((buf[offset + ref.numel():] == 0xEE).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_quantizer_marks_blocks_with_nan_or_inf(dtype):
    """A NaN or an infinity in a block gives scale byte 255 (E8M0's NaN) and codes 0, bit-exact against the oracle;
    read back through the reference's dequantisation rule the block is NaN, every other block is untouched, and a
    GEMM on it returns NaN for the row instead of finite numbers."""
    rows, K, N = 40, 512, 256
    g = torch.Generator().manual_seed(31)
    x = torch.randn(rows, K, generator=g)
    planted = {(1, 40): float("nan"), (2, 70): float("-inf"), (3, 0): float("inf"), (39, 511): float("nan"), (5, 100): float("inf")}
    x[5, 101] = float("nan")  # both kinds in one block
    for (r, k), v in planted.items():
        x[r, k] = v
    x = x.to(dtype)
    q, s, packed = wb.quantize_mxfp4(x.to(DEV))
    eq, es = orc.quantize_mxfp4(x.float())
    assert torch.equal(s.cpu(), es) and torch.equal(q.cpu(), eq)
    assert torch.equal(packed.data.cpu(), orc.pack_scales(es))
    bad = torch.zeros(rows, K // 32, dtype=torch.bool)
    for (r, k) in planted:
        bad[r, k // 32] = True
    assert torch.equal(s.cpu() == 255, bad)
    deq = orc.dequant_mxfp4(q.cpu(), s.cpu()).reshape(rows, K // 32, 32)
    assert torch.equal(torch.isnan(deq).all(dim=2), bad) and torch.equal(torch.isnan(deq).any(dim=2), bad)
    w, w_s = orc.quantize_mxfp4(torch.randn(N, K, generator=g))
    c = torch.zeros(rows, N, dtype=torch.float32, device=DEV)
    ops.scaled_gemm_packed(q, packed, w.to(DEV), ops.repack_scales(w_s.to(DEV)), c)
    nan_rows = bad.any(dim=1)
    assert torch.equal(torch.isnan(c).all(dim=1).cpu(), nan_rows) and torch.equal(torch.isnan(c).any(dim=1).cpu(), nan_rows)


def test_weight_scale_cache_belongs_to_the_tensor_not_the_address():
    """A new scale tensor that the allocator puts at a freed tensor's address must be repacked, an in-place write
    must be seen, and drop_cached_weights forgets a packing that a raw write made stale."""
    M, N, K = 64, 256, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=11)
    tpl, options = wb.templates.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, tpl)
    ad, asd, bd = a.to(DEV), a_s.to(DEV), b.to(DEV)
    c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    s1 = b_s.to(DEV)
    ptr = s1.data_ptr()
    gemm(ad, asd, bd, s1, c)
    check(c, a, a_s, b, b_s)
    del s1
    other = (b_s.to(torch.int16) + 1).clamp(max=131).to(torch.uint8)
    s2 = other.to(DEV)  # same shape: the caching allocator hands the freed block out again
    if s2.data_ptr() != ptr:
        pytest.skip("the allocator did not reuse the address")
    gemm(ad, asd, bd, s2, c)
    check(c, a, a_s, b, other)
    s2.copy_(b_s.to(DEV))  # in-place write: version counter moves
    gemm(ad, asd, bd, s2, c)
    check(c, a, a_s, b, b_s)
    # a write the version counter does not see (here through a detached alias of the memory)
    alias = torch.as_strided(s2.detach().view(-1).data, s2.shape, s2.stride())
    version = s2._version
    alias.data.copy_(other.to(DEV))
    if s2._version == version:
        gemm.drop_cached_weights(s2)
    gemm(ad, asd, bd, s2, c)
    check(c, a, a_s, b, other)


def test_mxfp4_linear_module_matches_oracle():
    torch.manual_seed(5)
    N, K = 768, 1024
    w = torch.randn(N, K) * 0.02
    x = torch.randn(3, 50, K)
    layer = wb.MXFP4Linear.from_float(w.to(DEV), output_dtype=torch.bfloat16)
    y = layer(x.to(DEV))
    assert y.shape == (3, 50, N) and y.dtype == torch.bfloat16
    wq, ws = orc.quantize_mxfp4(w)
    xq, xs = orc.quantize_mxfp4(x.reshape(-1, K))
    assert torch.equal(layer.weight_codes.cpu(), wq) and torch.equal(layer.weight_scales.cpu(), ws)
    check_bf16(y.reshape(-1, N), orc.scaled_gemm(xq, xs, wq, ws))


def test_mxfp4_linear_decode_batch_uses_the_balanced_packing():
    """A layer wide enough for the whole-tile decode kernel: small batches read the per-tile packing, large ones the usual
    one, both match the oracle."""
    torch.manual_seed(6)
    N, K = 28672, 256
    w = torch.randn(N, K) * 0.02
    layer = wb.MXFP4Linear.from_float(w.to(DEV), output_dtype=torch.bfloat16)
    wq, ws = orc.quantize_mxfp4(w)
    for rows in (4, 200, 4):
        x = torch.randn(rows, K)
        y = layer(x.to(DEV))
        xq, xs = orc.quantize_mxfp4(x)
        check_bf16(y, orc.scaled_gemm(xq, xs, wq, ws))
    assert layer._packed_decode.tile_rows == ops.decode_tile_rows(N) and layer._packed.tile_rows == 128
    ops.check_device_status()


def test_host_pipelined_gemm_on_pinned_buffers():
    """Five calls through the three-stream host pipeline with three device buffer sets: every result
    must belong to its own call's operands (no buffer reused before its result left the device)."""
    from wave_b200.host_pipeline import HostScaledGemm
    M, N, K = 200, 384, 512
    pipe = HostScaledGemm(M, N, K, wb.bf16, device=DEV, depth=3)
    problems = [random_problem(M, N, K, seed=80 + i) for i in range(5)]
    pinned = [[t.pin_memory() for t in p] for p in problems]
    outs = [torch.empty(M, N, dtype=torch.bfloat16).pin_memory() for _ in problems]
    for (a, a_s, b, b_s), c in zip(pinned, outs):
        pipe.submit(a, a_s, b, b_s, c)
    pipe.drain()
    for (a, a_s, b, b_s), c in zip(problems, outs):
        check_bf16(c, orc.scaled_gemm(a, a_s, b, b_s))
    with pytest.raises(ValueError, match="pinned"):
        pipe.submit(*problems[0], outs[0])
    ops.check_device_status()


# ---------------------------------------------------------------------------------------------
# the reference's own test shapes, and a seeded sweep of odd shapes
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("shape", [(1024, 1024, 8192), (1024, 1600, 8192), (1024, 1920, 8192), (1024, 3072, 8192)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_reference_macrotile_shapes_seed5(shape, out_dtype):
    """Shapes of testScaledGemmMXFP4ManualDoubleBuf / ...PreshuffleMacrotiles / ...8WavePingpong
    (wave_gemm_mxfp_test.py:637-680, 778-1085, 1088-1260), inputs from the reference's seed-5 generator,
    compared as the reference compares (default assert_close) and with this library's tolerances."""
    x, w, xs, ws = orc.generate_gemm_afp4wfp4_inputs(shape)
    w_t = w.T.contiguous()
    ref = orc.torch_scaled_gemm_mxfp4(x, w, xs, ws)
    kernel, options = wb.get_tagged_mxfp4_gemm_preshuffle_b(shape, (128, 256, 256), wave_shape=(1, 4),
                                                            output_dtype=wb.TORCH_DTYPE_TO_WAVE[out_dtype])
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel, wb.get_mxfp4_asymmetric_schedule())
    out = torch.zeros(shape[0], shape[1], dtype=out_dtype, device=DEV)
    gemm(x.to(DEV), wb.e8m0_shuffle(xs.to(DEV)), wb.b_preshuffle(w_t.to(DEV)), wb.e8m0_shuffle(ws.to(DEV)), out)
    torch.testing.assert_close(ref, out.cpu(), check_dtype=False)
    check(out, x, xs, w_t, ws, ref=ref)


def test_seeded_sweep_of_odd_shapes():
    """40 random (M, N, K) with K a multiple of 32 and nothing else aligned, automatic path choice,
    alternating output types; scales over a wider range than the fixed tests."""
    rng = torch.Generator().manual_seed(2024)
    for i in range(40):
        M = int(torch.randint(1, 700, (1,), generator=rng))
        N = int(torch.randint(1, 900, (1,), generator=rng))
        K = 32 * int(torch.randint(1, 40, (1,), generator=rng))
        a, a_s, b, b_s = random_problem(M, N, K, seed=1000 + i, lo=118, hi=136)
        out_dtype = torch.float32 if i % 2 else torch.bfloat16
        kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.TORCH_DTYPE_TO_WAVE[out_dtype])
        c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
        wb.wave_compile(options, kernel)(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
        ref = orc.scaled_gemm(a, a_s, b, b_s)
        if out_dtype == torch.float32:
            try:
                check_f32(c, a, a_s, b, b_s, ref)
            except AssertionError as e:
                raise AssertionError(f"shape {(M, N, K)} f32: {e}") from e
        else:
            # With scales spread over 18 binades some outputs are sums that cancel to far below their
            # terms; there the f32 bound (which has an absolute part) governs, and the bf16 result may
            # sit more than one ulp from the rounded reference. Everywhere else: 1 ulp.
            ulp = orc.bf16_ulp_distance(c, ref)
            tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s), orc.dequant_mxfp4(b, b_s), ref, K)
            half_ulp = ref.abs() * 2.0 ** -8
            bad = (ulp > 1) & ~((c.float().cpu() - ref).abs() <= tol + half_ulp)
            assert not bool(bad.any()), f"shape {(M, N, K)} bf16: {int(bad.sum())} outside both bounds"
            assert float((ulp > 1).float().mean()) < 1e-3, f"shape {(M, N, K)} bf16: too many entries beyond 1 ulp"
        ops.check_device_status()


def test_nan_scale_propagates_like_the_reference():
    """Scale code 255 is NaN in the reference (mxfp_utils.py:92-94): the rows and columns it touches are
    NaN in the output, everything else is unaffected."""
    M, N, K = 64, 96, 256
    a, a_s, b, b_s = random_problem(M, N, K, seed=3)
    a_s[5, 2] = 255
    b_s[7, 0] = 255
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    c = run(a, a_s, b, b_s, torch.float32).cpu()
    assert torch.equal(c.isnan(), ref.isnan()) and bool(ref.isnan()[5].all()) and bool(ref.isnan()[:, 7].all())
    ok = ~ref.isnan()
    tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s).nan_to_num(0), orc.dequant_mxfp4(b, b_s).nan_to_num(0), ref.nan_to_num(0), K)
    assert bool(((c - ref).abs()[ok] <= tol[ok]).all())


def test_cuda_graph_replay_of_a_decode_call():
    from wave_b200.graphs import GraphedScaledGemm
    M, N, K = 16, 2048, 1024
    a, a_s, b, b_s = random_problem(M, N, K, seed=91)
    a2, a2_s, _, _ = random_problem(M, N, K, seed=92)
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)
    ad, asd, bd, bsd = a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV)
    c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    g = GraphedScaledGemm(gemm, ad, asd, bd, bsd, c)
    g.replay()
    check_bf16(c, orc.scaled_gemm(a, a_s, b, b_s))
    ad.copy_(a2.to(DEV)); asd.copy_(a2_s.to(DEV))          # new activations in the same buffers
    g.replay()
    check_bf16(c, orc.scaled_gemm(a2, a2_s, b, b_s))
    ops.check_device_status()


def test_packed_weight_scales_of_a_captured_call_outlive_their_eviction():
    """One kernel object over more weights than its cache holds, captured into one graph: every captured call keeps the packing it was
    given, also after later calls have evicted it and `drop_cached_weights` has emptied the cache."""
    M, N, K, n = 16, 2048, 1024, 4
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    gemm._weight_scales.capacity = 2
    probs = [random_problem(M, N, K, seed=40 + i) for i in range(n)]
    dev = [[t.to(DEV) for t in p] for p in probs]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in probs]
    side, graph = torch.cuda.Stream(DEV), torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        for p, c in zip(dev, outs):
            gemm(*p, c)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        for p, c in zip(dev, outs):
            gemm(*p, c)
    assert len(gemm._weight_scales._entries) <= 2 and len(gemm._weight_scales._captured) == n
    for p, ref, c in zip(dev, probs, outs):  # before any replay: a packing made in the capture holds nothing yet
        gemm(*p, c)
        check(c, *ref)
    gemm.drop_cached_weights()
    blocks = [torch.full((ops.packed_scale_bytes(N, K),), 255, dtype=torch.uint8, device=DEV) for _ in range(16)]
    for c in outs:
        c.fill_(float("nan"))
    graph.replay()
    for p, c in zip(probs, outs):
        check(c, *p)
    assert all(bool((t == 255).all()) for t in blocks)


def test_graphed_gemm_keeps_the_kernel_object_alive():
    """The graph holds addresses of memory that belongs to the kernel object (workspace, scratch, packed weight scales): a graph whose
    maker dropped that object still has it, and gives the same result after its memory could have been handed out again."""
    import gc
    import weakref
    from wave_b200.graphs import GraphedScaledGemm
    M, N, K = 16, 4096, 1024
    a, a_s, b, b_s = random_problem(M, N, K, seed=12)
    dev = [t.to(DEV) for t in (a, a_s, b, b_s)]
    c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)

    def make():
        kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
        gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
        return GraphedScaledGemm(gemm, *dev, c), weakref.ref(gemm)

    graphed, gemm = make()
    gc.collect()
    assert gemm() is not None
    blocks = [torch.full((n,), 255, dtype=torch.uint8, device=DEV) for n in (1 << 14, 1 << 18, 1 << 20, 1 << 22) for _ in range(4)]
    c.fill_(float("nan"))
    graphed.replay()
    check(c, a, a_s, b, b_s)
    assert all(bool((t == 255).all()) for t in blocks)
    del graphed
    gc.collect()
    assert gemm() is None


def test_bounded_wait_reports_timeout_and_context_stays_usable():
    """A wait that nothing satisfies gives up after its limit, the kernel ends normally, the status word
    carries the code, and the next GEMM on the same context is correct."""
    lib = _lib.load()
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.wb200_selftest_wait_timeout(2_000_000, stream))  # ~1 ms
    with pytest.raises(_lib.DeviceTimeoutError, match="wait 7"):
        ops.check_device_status()
    ops.check_device_status()  # the word was cleared
    assert lib.wb200_selftest_wait_timeout(10 ** 12, stream) == _lib.WB200_ERR_INVALID_ARG
    a, a_s, b, b_s = random_problem(256, 256, 512, seed=17)
    check(run(a, a_s, b, b_s, torch.float32), a, a_s, b, b_s)


def test_single_row_operands_with_arbitrary_size_one_stride():
    """M = 1 through the reference's generator: `x_scales.T.contiguous()` of a [K/32, 1] tensor is a
    [1, K/32] tensor whose row stride is 1, not K/32."""
    shape = (1, 512, 1024)
    x, w, xs, ws = orc.generate_gemm_afp4wfp4_inputs(shape)
    assert xs.shape == (1, 32)
    w_t = w.T.contiguous()
    kernel, options = wb.get_tagged_mxfp4_gemm(shape, output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)
    c = torch.empty(1, 512, dtype=torch.bfloat16, device=DEV)
    xs_dev = xs.to(DEV).T.contiguous().T  # keeps the odd stride on the device
    for _ in range(2):  # first call: checked path; second: remembered-signature path
        gemm(x.to(DEV), xs_dev, w_t.to(DEV), ws.to(DEV), c)
        check_bf16(c, orc.torch_scaled_gemm_mxfp4(x, w, xs, ws))


def test_broadcasted_scale_gemm_as_the_reference_tests_it():
    """testBroadcastedScaleGemmMXFP4 (tests/kernel/wave_gemm_mxfp_test.py:594-634): a_scale is the first
    column of the generated scales, shape [M]; the oracle gets it repeated along K."""
    shape = (512, 512, 512)
    kernel, hyper = wb.get_broadcasted_scale_gemm_mxfp4(shape, wb.ScaledMMAType.F32_16x16x128_F8F6F4)
    options = wb.WaveCompileOptions(subs=hyper, canonicalize=True, schedule=wb.SchedulingType.NONE)
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    x, w, x_scales, w_scales = orc.generate_gemm_afp4wfp4_inputs(shape)
    compact = x_scales[:, 0].contiguous()
    out = torch.zeros(shape[0], shape[1], dtype=torch.float32, device=DEV)
    w_t = w.T.contiguous()
    gemm(x.to(DEV), compact.to(DEV), w_t.to(DEV), w_scales.to(DEV), out)
    full = compact.view(-1, 1).repeat(1, x_scales.shape[-1]).contiguous()
    torch_out = orc.torch_scaled_gemm_mxfp4(x, w, full, w_scales)
    torch.testing.assert_close(torch_out, out.cpu(), check_dtype=False)
    check(out, x, full, w_t, w_scales, ref=torch_out)
    # the packed form is bit-identical to packing the repeated scales, also for a strided, ragged source
    wide = torch.randint(0, 256, (300, 3), dtype=torch.uint8)
    got = ops.repack_scales_broadcast(wide.to(DEV)[:, 1], 1184)
    assert torch.equal(got.data.cpu(), orc.pack_scales(wide[:, 1:2].repeat(1, 1184 // 32).contiguous()))
    with pytest.raises(ValueError):
        gemm(x.to(DEV), x_scales.to(DEV), w_t.to(DEV), w_scales.to(DEV), out)


@pytest.mark.parametrize("ways", [8, 2])
def test_config5_one_shard_of_the_sharded_gemm_bf16_sampled(ways):
    """M = 16384, N = 53248, K = 16384 sharded over `ways` GPUs by rows of b: one GPU's shard
    (N / ways = 6656 or 26624 rows) at full size. Operands are seeded f32 N(0, 1) matrices (seeds 1005 / 2005)
    quantised on the GPU (the quantiser is bit-exact against the oracle's, tested above); the oracle is evaluated for
    sampled rows of a against sampled row blocks of the shard, and the whole shard is checked through the exact
    doubling property. Bar: 1 bf16 ulp of the rounded f32 reference. An entry further away passes only where the f32
    bound holds (a sum that cancels far below its terms, so that the accumulation order moves it across more than one
    bf16 step); such entries are counted and reported, and there may be at most one in ten thousand."""
    M, N, K = 16384, 53248, 16384
    n_shard = N // ways
    assert n_shard % 256 == 0
    g = torch.Generator(device=DEV).manual_seed(1005)
    a, a_s, _ = ops.quantize_mxfp4(torch.randn(M, K, device=DEV, generator=g, dtype=torch.float32), want_packed=False)
    g.manual_seed(2005)
    b, b_s, _ = ops.quantize_mxfp4(torch.randn(n_shard, K, device=DEV, generator=g, dtype=torch.float32), want_packed=False)
    kernel, options = wb.get_tagged_mxfp4_gemm((M, n_shard, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)
    c = torch.empty(M, n_shard, dtype=torch.bfloat16, device=DEV)
    gemm(a, a_s, b, b_s, c)
    rows = torch.arange(0, M, 683, device=DEV)
    escaped = checked = 0
    for n0 in (0, (n_shard // 2) // 256 * 256 + 128, n_shard - 1024):
        ref = orc.scaled_gemm(a[rows].cpu(), a_s[rows].cpu(), b[n0:n0 + 1024].cpu(), b_s[n0:n0 + 1024].cpu())
        got = c[rows][:, n0:n0 + 1024].contiguous()
        ulp = orc.bf16_ulp_distance(got, ref)
        tol = orc.f32_tolerance(orc.dequant_mxfp4(a[rows].cpu(), a_s[rows].cpu()),
                                orc.dequant_mxfp4(b[n0:n0 + 1024].cpu(), b_s[n0:n0 + 1024].cpu()), ref, K)
        within_f32 = (got.float().cpu() - ref).abs() <= tol
        failed = (ulp > 1) & ~within_f32
        assert not bool(failed.any()), f"{int(failed.sum())} entries beyond 1 bf16 ulp and beyond the f32 bound (max {int(ulp.max())} ulp)"
        escaped += int(((ulp > 1) & within_f32).sum())
        checked += ulp.numel()
    if escaped:
        import warnings
        warnings.warn(f"config 5, {ways}-way shard: {escaped} of {checked} sampled entries are more than 1 bf16 ulp from the "
                      "rounded reference and pass by the f32 bound")
    assert escaped * 10000 <= checked
    c2 = torch.empty_like(c)
    gemm(a, a_s + 1, b, b_s, c2)
    assert torch.equal((c.float() * 2).to(torch.bfloat16), c2)
    ops.check_device_status()


@pytest.mark.parametrize("shape", [(512, 512, 16000), (256, 512, 4096), (1000, 300, 8192), (300, 260, 2560), (2048, 512, 16000)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_split_k_tile_path(shape, out_dtype):
    """Few output tiles and a long K (the small-N end of the reference's benchmark shapes,
    perf/mxfp4_shapes_macrotiles.csv): K slices x tiles in one launch, partial products added in slice order."""
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K, lo=125, hi=129)
    ad, bd = a.to(DEV), b.to(DEV)
    asp, bsp = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, asp, bd, bsp, c, _lib.PATH_TILE_SPLITK)
    check(c, a, a_s, b, b_s, ref=ref)
    auto = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops.scaled_gemm_packed(ad, asp, bd, bsp, auto)  # the automatic choice (split-K from three slices up)
    check(auto, a, a_s, b, b_s, ref=ref)
    if out_dtype == torch.float32:  # the split-K templates' contract: add into a caller-initialised c
        base = torch.randn(M, N)
        acc = base.to(DEV)
        ops.scaled_gemm_packed(ad, asp, bd, bsp, acc, _lib.PATH_TILE_SPLITK | _lib.ACCUMULATE)
        tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s), orc.dequant_mxfp4(b, b_s), ref, K)
        assert bool(((acc.cpu() - (ref + base)).abs() <= tol + 1e-6 * base.abs()).all())
    ops.check_device_status()


def test_split_k_is_the_automatic_choice_under_graph_capture_only():
    """Eager Python calls keep the plain tile path (the split-K launch costs more host time than it saves on
    the GPU for a slow host); a call captured into a CUDA graph takes split-K. Both match the oracle; the
    captured one equals the forced split-K result bit for bit."""
    M, N, K = 512, 512, 8192
    a, a_s, b, b_s = random_problem(M, N, K, seed=77, lo=125, hi=129)
    ad, bd = a.to(DEV), b.to(DEV)
    asp, bsp = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    forced = torch.empty(M, N, dtype=torch.float32, device=DEV)
    plain = torch.empty_like(forced)
    eager = torch.empty_like(forced)
    captured = torch.empty_like(forced)
    ops.scaled_gemm_packed(ad, asp, bd, bsp, forced, _lib.PATH_TILE_SPLITK)
    ops.scaled_gemm_packed(ad, asp, bd, bsp, plain, _lib.PATH_TILE_2CTA | _lib.TILE_N128)
    ops.scaled_gemm_packed(ad, asp, bd, bsp, eager)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.scaled_gemm_packed(ad, asp, bd, bsp, captured)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager, plain) and torch.equal(captured, forced)
    check(captured, a, a_s, b, b_s)
    check(eager, a, a_s, b, b_s)


def test_split_k_tile_path_refuses_what_it_cannot_do():
    a, a_s, b, b_s = random_problem(4096, 4096, 1024, seed=1)
    c = torch.empty(4096, 4096, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(RuntimeError):  # plenty of tiles: not a split-K shape
        ops.scaled_gemm_packed(a.to(DEV), ops.repack_scales(a_s.to(DEV)), b.to(DEV), ops.repack_scales(b_s.to(DEV)), c,
                               _lib.PATH_TILE_SPLITK)


@pytest.mark.parametrize("shape", [(16, 4096, 2048), (100, 1000, 992), (512, 768, 1024)])
def test_overlap_previous_chain_gives_the_same_bits(shape):
    """Back-to-back calls flagged WB200_OVERLAP_PREVIOUS (each launched as a programmatic dependent of the one
    before it, sharing scratch and workspace) against the same calls launched one after the other."""
    M, N, K = shape
    kernel, options = wb.get_tagged_mxfp4_gemm(shape, output_dtype=wb.bf16)
    plain = wb.wave_compile(wb.set_default_run_config(options), kernel)
    kernel2, options2 = wb.get_tagged_mxfp4_gemm(shape, output_dtype=wb.bf16)
    options2.overlap_previous = True
    chained = wb.wave_compile(wb.set_default_run_config(options2), kernel2)
    probs = [random_problem(M, N, K, seed=500 + i) for i in range(4)]
    dev_probs = [[t.to(DEV) for t in p] for p in probs]
    ref_out = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in probs]
    for p, c in zip(dev_probs, ref_out):
        plain(p[0], p[1], p[2], p[3], c)
        torch.cuda.synchronize()
    outs = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in probs]
    for rep in range(3):  # no synchronisation between the calls
        for p, c in zip(dev_probs, outs):
            chained(p[0], p[1], p[2], p[3], c)
    torch.cuda.synchronize()
    for c, r in zip(outs, ref_out):
        assert torch.equal(c.view(torch.int16), r.view(torch.int16))
    check_bf16(outs[0], orc.scaled_gemm(*probs[0]))
    ops.check_device_status()


@pytest.mark.parametrize("strided", [False, True])
def test_overlap_previous_waits_for_the_weight_scales_the_call_packs_itself(strided):
    """A call that has to pack its weight's scales puts a kernel that writes them in front of its GEMM: that call is not launched as
    the kernel's early dependent, the next one is. Both through the remembered plan and through the general form (strided a)."""
    M, N, K = 16, 28672, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=3)
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    options.overlap_previous = True
    gemm = wb.wave_compile(wb.set_default_run_config(options), kernel)
    lib, seen = _lib.load(), []

    class Recorder:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            if not name.startswith("wb200_mxfp4_gemm") or name.endswith("bytes"):
                return fn
            return lambda *args: (seen.append(args[-2]), fn(*args))[1]

    gemm._lib = Recorder()
    ad = a.to(DEV)
    if strided:
        wide = torch.zeros(M, K // 2 + 16, dtype=torch.uint8, device=DEV)
        wide[:, :K // 2] = ad
        ad = wide[:, :K // 2]
    bd, a_sd, b_sd = b.to(DEV), a_s.to(DEV), b_s.to(DEV)
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(_lib, "load", lambda: gemm._lib)
        for call in range(3):
            if call == 2:
                b_sd.copy_(b_s)  # a new version: packed again
            c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
            gemm(ad, a_sd, bd, b_sd, c)
            check(c, a, a_s, b, b_s)
    assert [bool(f & _lib.OVERLAP_PREVIOUS) for f in seen] == [False, True, False]


def test_a_weight_quantised_two_launches_ahead_of_an_overlapping_gemm():
    """quantise w -> GEMM on another weight -> GEMM on w, both GEMMs flagged WB200_OVERLAP_PREVIOUS: the kernel before the second
    GEMM does not write w, so that GEMM may load w at once, and the quantiser has to be done by then. w's memory holds the
    other of two weights before every round, so a value read too early is a wrong one."""
    N, K, M = 16384, 8192, 16
    lib, g = _lib.load(), torch.Generator(device=DEV).manual_seed(5)
    ws = [torch.randn(N, K, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2)]
    q, pk = torch.empty(N, K // 2, dtype=torch.uint8, device=DEV), torch.empty(ops.packed_scale_bytes(N, K), dtype=torch.uint8, device=DEV)
    a, _, a_sf = ops.quantize_mxfp4(torch.randn(M, K, generator=g, device=DEV))
    q1, _, sf1 = ops.quantize_mxfp4(torch.randn(1024, K, generator=g, device=DEV))
    c1, w_sf = torch.empty(M, 1024, dtype=torch.bfloat16, device=DEV), ops.PackedScales(pk, N, K)

    def quantise(w):
        _lib.check(lib.wb200_quantize_mxfp4(w.data_ptr(), _lib.WB200_BF16, K, N, K, q.data_ptr(), None, pk.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))

    refs = []
    for w in ws:
        quantise(w)
        torch.cuda.synchronize()
        refs.append(torch.empty(M, N, dtype=torch.bfloat16, device=DEV))
        ops.scaled_gemm_packed(a, a_sf, q, w_sf, refs[-1])
    outs = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(6)]
    for i, c in enumerate(outs):  # no synchronisation in between
        quantise(ws[i & 1])
        ops.scaled_gemm_packed(a, a_sf, q1, sf1, c1, _lib.OVERLAP_PREVIOUS)
        ops.scaled_gemm_packed(a, a_sf, q, w_sf, c, _lib.OVERLAP_PREVIOUS)
    torch.cuda.synchronize()
    for i, c in enumerate(outs):
        assert torch.equal(c.view(torch.int16), refs[i & 1].view(torch.int16))
    ops.check_device_status()


def test_run_bench_option_reports_kernel_time(tmp_path):
    """options.run_bench: after the call the kernel is timed on the device and the report goes to
    benchmark_results_file (the reference hands its module to a benchmark tool, compile.py:317-329)."""
    import json
    a, a_s, b, b_s = random_problem(128, 256, 512, seed=3)
    kernel, options = wb.get_tagged_mxfp4_gemm((128, 256, 512), output_dtype=wb.bf16)
    options.run_bench, options.benchmark_batch_size, options.benchmark_repetitions = True, 5, 3
    options.benchmark_results_file = str(tmp_path / "bench.json")
    gemm = wb.wave_compile(options, kernel)
    c = torch.empty(128, 256, dtype=torch.bfloat16, device=DEV)
    gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), c)
    check(c, a, a_s, b, b_s)
    rep = json.loads((tmp_path / "bench.json").read_text())["benchmarks"][0]
    assert rep["time_unit"] == "us" and rep["iterations"] == 3 and 0 < rep["min_time"] <= rep["real_time"] < 1e5


@pytest.mark.parametrize("shape", [(129, 128, 10240), (512, 2048, 16000), (300, 1000, 10016), (700, 900, 16384), (512, 512, 12000),
                                   (1024, 1030, 10272)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_split_k_inside_a_cluster(shape, out_dtype):
    """Few output tiles and K >= 40 K blocks without a workspace: the slices of a tile run on the CTA pairs of one cluster. One
    tile and the most that 2, 3 and 4 slices take; ragged M, N and K, C with an unaligned row pitch, accumulation, and the
    same bits on every run."""
    M, N, K = shape
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K, lo=125, hi=129)
    ad, bd = a.to(DEV), b.to(DEV)
    asp, bsp = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    wide = torch.full((M, N + 3), float("nan"), dtype=out_dtype, device=DEV)
    c = wide[:, 1:N + 1]
    ops.scaled_gemm_packed(ad, asp, bd, bsp, c)
    check(c.contiguous(), a, a_s, b, b_s, ref=ref)
    assert bool(wide[:, 0].isnan().all()) and bool(wide[:, N + 1:].isnan().all())
    again = torch.empty(M, N, dtype=out_dtype, device=DEV)
    for _ in range(3):
        ops.scaled_gemm_packed(ad, asp, bd, bsp, again)
        assert torch.equal(again, c)
    if out_dtype == torch.float32:
        base = torch.randn(M, N, generator=torch.Generator().manual_seed(M))
        acc = base.to(DEV)
        ops.scaled_gemm_packed(ad, asp, bd, bsp, acc, _lib.ACCUMULATE)
        tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s), orc.dequant_mxfp4(b, b_s), ref, K)
        assert bool(((acc.cpu() - (ref + base)).abs() <= tol + 1e-6 * base.abs()).all())
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K", [(1, 640, 992), (16, 28672, 256), (33, 1000, 1184), (64, 19072, 288), (100, 28672 - 40, 512), (128, 4096, 2080),
                                   (129, 512, 32), (300, 700, 1184), (1000, 384, 4128), (2048, 4096, 512), (2050, 8192, 288)])
@pytest.mark.parametrize("offset,extra", [(0, 0), (8, 8), (3, 5)])
def test_row_major_activation_scales_give_the_bits_of_packed_ones(M, N, K, offset, extra):
    """The call that takes a_scale row-major against the same GEMM on scales packed beforehand, for every path of the call: the sizes at
    which it packs them itself ahead of the GEMM (nearly all of these; the next test is for the kernels that take them as they
    are), K blocks that end inside a stage, rows that end inside a tile, row pitches and bases of any alignment."""
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K + offset)
    wide = torch.full((M, offset + K // 32 + extra), 255, dtype=torch.uint8, device=DEV)
    view = wide[:, offset:offset + K // 32]
    view.copy_(a_s.to(DEV))
    kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(options, kernel)
    ad, bd, bsd = a.to(DEV), b.to(DEV), b_s.to(DEV)
    c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    gemm(ad, view, bd, bsd, c)
    ref = torch.full_like(c, float("nan"))
    h = ops.decode_tile_rows(N) if M <= 128 else 128
    ops.scaled_gemm_packed(ad, ops.repack_scales(a_s.to(DEV)), bd, ops.repack_scales(bsd, tile_rows=h), ref)
    assert torch.equal(c.view(torch.int16), ref.view(torch.int16))
    check(c, a, a_s, b, b_s)
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K,pad,path", [
    (16, 28672, 288, 7, 0), (32, 28672, 2336, 7, 0), (1, 28672, 4096, 0, 0), (5, 57344, 2816, 8, 0),  # whole tiles: one and more rounds
    (17, 19000, 3104, 7, 0), (32, 18816 + 128, 512, 0, 0),
    (16, 9472, 4128, 7, 0), (3, 14336, 4096, 0, 0), (16, 4096, 10272, 7, 0),  # K split
    (17, 1000, 2336, 7, _lib.PATH_SKINNY), (32, 640, 8192, 0, _lib.PATH_SKINNY), (1, 128, 32, 7, _lib.PATH_SKINNY), (30, 300, 12576, 15, _lib.PATH_SKINNY),
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_decode_kernels_take_row_major_scales_as_they_are(M, N, K, pad, path, out_dtype):
    """The warp that brings row-major scales into the stages, in both decode kernels: fewer and more K blocks than ring stages, runs over
    several tiles, the last K blocks of a row (K / 32 not a multiple of 8 with a padded pitch), fewer rows than lanes. Bits of
    the same GEMM on packed scales, the oracle's values, and a scratch that stays as it was: no repack kernel ran."""
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K)
    pitch = (K // 32 + pad) // 8 * 8 if pad else K // 32
    assert pitch >= K // 32 and pitch % 8 == 0
    wide = torch.full((M + 1, pitch), 255, dtype=torch.uint8, device=DEV)
    view = wide[1:, :K // 32]
    view.copy_(a_s.to(DEV))
    lib, h = _lib.load(), ops.decode_tile_rows(N)
    if path:
        h = 128
    flags = path | _lib.B_TILE_ROWS(h)
    b_sf, ad, bd = ops.repack_scales(b_s.to(DEV), tile_rows=h), a.to(DEV), b.to(DEV)
    scratch = torch.full((ops.packed_scale_bytes(M, K),), 0xEE, dtype=torch.uint8, device=DEV)
    ws_bytes = int(lib.wb200_mxfp4_gemm_workspace_bytes(M, N, K))
    c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    for _ in range(2):
        _lib.check(lib.wb200_mxfp4_gemm_repack_a(M, N, K, ad.data_ptr(), view.data_ptr(), pitch, scratch.data_ptr(), bd.data_ptr(),
                                                 b_sf.data.data_ptr(), c.data_ptr(), ops._DTYPE_CODE[out_dtype], N,
                                                 ops._workspace(ad.device, ws_bytes).data_ptr(), ws_bytes, flags,
                                                 torch.cuda.current_stream().cuda_stream))
    assert bool((scratch == 0xEE).all())
    ref = torch.full_like(c, float("nan"))
    ops.scaled_gemm_packed(ad, ops.repack_scales(a_s.to(DEV)), bd, b_sf, ref, path)
    bits = torch.int16 if out_dtype == torch.bfloat16 else torch.int32
    assert torch.equal(c.view(bits), ref.view(bits))
    check(c, a, a_s, b, b_s)


@pytest.mark.parametrize("N,K", [(128, 256), (500, 1024), (1024, 8192), (1030, 12288), (4096, 4064), (9472, 4096), (9601, 4096), (18816, 512),
                                 (14336, 4096), (2048, 16000), (4096, 10240), (5803, 5376), (8192, 8192), (11001, 4096)])
@pytest.mark.parametrize("M", [1, 16, 17, 32, 64, 128])
def test_decode_calls_with_few_weight_tiles(M, N, K):
    """M <= 128 with fewer 128-row weight tiles than SMs: the K-split kernel, the two tile kernels or a cluster per tile, by M, the
    size of the weight, that of the activations and the alignment of C's rows; either side of every line of that rule. Same call as a user's (AUTO, with a workspace)."""
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K)
    ad, bd = a.to(DEV), b.to(DEV)
    a_sf, b_sf = ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    for out_dtype in (torch.bfloat16, torch.float32):
        c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
        ops.scaled_gemm_packed(ad, a_sf, bd, b_sf, c)
        check(c, a, a_s, b, b_s, ref=ref)
    base = torch.randn(M, N, generator=torch.Generator().manual_seed(N))
    acc = base.to(DEV)
    ops.scaled_gemm_packed(ad, a_sf, bd, b_sf, acc, _lib.ACCUMULATE)
    tol = orc.f32_tolerance(orc.dequant_mxfp4(a, a_s), orc.dequant_mxfp4(b, b_s), ref, K)
    assert bool(((acc.cpu() - (ref + base)).abs() <= tol + 1e-6 * base.abs()).all())
    ops.check_device_status()


@pytest.mark.parametrize("rows,N,K", [(1, 640, 416), (32, 28672, 256), (128, 1000, 992), (129, 512, 288), (1000, 4096, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_linear_in_one_call_gives_the_bits_of_quantiser_and_gemm(rows, N, K, dtype):
    """MXFP4Linear's single native call against wb200_quantize_mxfp4 followed by the GEMM, also for a column block of a wider x and
    for a transposed x, which is copied."""
    g = torch.Generator().manual_seed(rows + N)
    layer = wb.MXFP4Linear.from_float((torch.randn(N, K, generator=g) * 0.02).to(DEV), output_dtype=dtype)
    wide = torch.randn(rows, K + 32, generator=g).to(dtype).to(DEV)
    for x in (wide[:, :K].contiguous(), wide[:, 16:K + 16], wide[:, :K].t().contiguous().t()):
        y = layer(x)
        q, _, sf = ops.quantize_mxfp4(x, want_rowmajor=False)
        ref = torch.empty(rows, N, dtype=dtype, device=DEV)
        ops.scaled_gemm_packed(q, sf, layer.weight_codes, layer._packed_decode if rows <= 128 else layer._packed, ref)
        assert torch.equal(y, ref)
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K,kind", [(8, 640, 416, "fp4"), (300, 512, 1024, "fp4"), (16, 1024, 512, "fp8"), (16, 1024, 512, "mixed")])
def test_a_repeated_call_follows_its_tensors(M, N, K, kind):
    """The second call with tensors of the same form is recognised in native code. It reads the tensors it is given (other activations, other
    weights, scales rewritten in place, another stream, a transposed operand, a wider output), and refuses what the first call would. Each
    result has the bits of a fresh kernel object's first call."""
    def operands(seed):
        g = torch.Generator().manual_seed(seed)
        if kind == "fp4":
            return [t.to(DEV) for t in random_problem(M, N, K, seed=seed)]
        x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
        b = ops.quantize_mxfp8(w, torch.float8_e4m3fn) if kind == "fp8" else ops.quantize_mxfp4(w)
        return [*ops.quantize_mxfp8(x, torch.float8_e4m3fn)[:2], *b[:2]]

    def compiled():
        if kind == "fp4":
            t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
        else:
            t, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4, "f8e4m3fn", wb.bf16,
                                                      weight_format="f4e2m1fn" if kind == "mixed" else None)
            options = wb.WaveCompileOptions(subs=subs)
        return wb.wave_compile(wb.set_default_run_config(options), t)

    gemm = compiled()
    wide = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device=DEV)

    def expect(args, c=None):
        c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) if c is None else c
        ref = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        gemm(*args, c)
        compiled()(*args, ref)
        assert torch.equal(c, ref)

    one, two = operands(1), operands(2)
    for args in (one, one, two, two, one[:2] + two[2:], one):
        expect(args)
    one[3].copy_(two[3])  # in place: the version counter moves
    expect(one)
    expect(one)
    for _ in range(2):
        expect(one, wide[:, :N])
        expect(one, wide[:, 1:N + 1])  # rows that are not 16-byte aligned
    assert bool((wide[:, N + 1:] == 7.0).all())
    bits = one[0].view(torch.uint8)
    expect([bits.t().contiguous().t().view(one[0].dtype), *one[1:]])
    torch.cuda.synchronize()
    side = torch.cuda.Stream(DEV)
    with torch.cuda.stream(side):
        expect(one)
        expect(two)
    side.synchronize()
    with torch.inference_mode():
        expect([one[0].clone(), *one[1:]])
    good = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    for bad in ([one[0][:-1], *one[1:], good], [one[0], one[1][:, :-1], *one[2:], good], [*one, good[:, :-1]], [*one, good.float()],
                [*one[:3], one[3][:-1], good], [one[0].cpu(), *one[1:], good], [*one[:2], one[2][:-1], one[3], good]):
        with pytest.raises(ValueError):
            gemm(*bad)
    gemm.drop_cached_weights()
    expect(one)
    ops.check_device_status()


def test_a_repeated_linear_call_follows_its_tensors():
    """MXFP4Linear: second and later calls, at several batch sizes, with strided, transposed, 1-D and 3-D inputs, on another stream, in a
    captured graph; each has the bits of the call that a new layer makes first."""
    N, K = 640, 416
    g = torch.Generator().manual_seed(1)
    layer = wb.MXFP4Linear.from_float((torch.randn(N, K, generator=g) * 0.02).to(DEV))
    wide = torch.randn(200, K + 32, generator=g).to(torch.bfloat16).to(DEV)

    def expect(x):
        y, ref = layer(x), wb.MXFP4Linear(layer.weight_codes, layer.weight_scales)(x)
        assert y.shape == (*x.shape[:-1], N) and torch.equal(y, ref)

    for _ in range(2):
        for x in (wide[:3, :K], wide[:200, 16:K + 16], wide[:8, :K].float(), wide[0, :K], wide[:6, :K].reshape(2, 3, K), wide[:, :K].t().contiguous().t()):
            expect(x)
        with torch.cuda.stream(torch.cuda.Stream(DEV)):
            expect(wide[:3, :K])
            torch.cuda.current_stream().synchronize()
    with pytest.raises(RuntimeError):
        layer(wide[:3, :K - 32])
    with pytest.raises(ValueError):
        layer(wide[:3, 1:K + 1])  # rows that are not 16-byte aligned
    x = wide[:4, :K].contiguous()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    x.copy_(wide[10:14, :K])
    graph.replay()
    assert torch.equal(y, layer(wide[10:14, :K]))
    ops.check_device_status()


@pytest.mark.parametrize("N,K", [(8, 32), (1000, 2048), (4096, 4096), (5803, 5376), (11001, 8192), (14336, 4096), (14335, 2080), (17800, 8192), (18900, 4096),
                                 (17408, 10240), (20480, 4096), (20483, 1024)])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 128])
def test_low_decode_tiles_match_the_usual_packing(M, N, K):
    """One low weight tile per SM, and several of them over a short K, in the template call: heights from 8 to 128, tiles that end past N, K
    that ends inside a stage, rows of C that are 16-byte aligned or not. Against the oracle (the bars of every decode kernel: one
    bf16 ulp, or the f32 bound) and the same call on the usual packing."""
    a, a_s, b, b_s = random_problem(M, N, K, seed=M + N + K)
    ad, asd, bd, bsd = a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV)
    ref = orc.scaled_gemm(a, a_s, b, b_s)
    for out_dtype in (torch.bfloat16, torch.float32):
        outs = []
        for tiled in (True, False):
            kernel, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.TORCH_DTYPE_TO_WAVE[out_dtype])
            options.decode_tiled_weight_scales = tiled
            c = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
            wb.wave_compile(options, kernel)(ad, asd, bd, bsd, c)
            outs.append(c)
        for c in outs:
            check(c, a, a_s, b, b_s, ref=ref)
        h = ops.decode_tile_rows_for(M, N, K, c_aligned=ops.rows_aligned(c))
        assert h % 8 == 0 and 8 <= h <= 128
    if h != 128 and N % 8 == 0:  # added into a C that holds values
        acc = torch.ones(M, N, device=DEV)
        ops.scaled_gemm_packed(ad, ops.repack_scales(asd), bd, ops.repack_scales(bsd, tile_rows=h), acc, _lib.ACCUMULATE)
        check(acc, a, a_s, b, b_s, ref=ref + 1.0)
    ops.check_device_status()


def test_linear_layer_first_used_at_another_decode_batch():
    """One layer at batch sizes that read different packings of its weight scales, in any order."""
    N, K = 14336, 512
    g = torch.Generator().manual_seed(3)
    w = torch.randn(N, K, generator=g) * 0.02
    wq, ws = orc.quantize_mxfp4(w)
    layer = wb.MXFP4Linear.from_float(w.to(DEV), output_dtype=torch.bfloat16)
    for rows in (128, 4, 128, 33, 200, 1):
        x = torch.randn(rows, K, generator=g)
        xq, xs = orc.quantize_mxfp4(x)
        check_bf16(layer(x.to(DEV)), orc.scaled_gemm(xq, xs, wq, ws))
    assert layer._packed.tile_rows == 128
    ops.check_device_status()


@pytest.mark.parametrize("captured", [False, True])
def test_calls_see_what_the_kernel_before_them_wrote(captured):
    """Every launch may become resident beside the kernel before it and waits for that kernel before it touches memory: operands,
    scales, weights and outputs that an ordinary kernel, or another call of the library, has written just before are the ones that are read,
    back to back and many times. Bits of the same calls with a synchronisation between all of them."""
    g = torch.Generator(device=DEV)
    cases = []
    for M, N, K in ((8, 4096, 512), (200, 512, 768), (16, 19456, 256), (300, 1024, 512)):
        b, b_s, b_sf = ops.quantize_mxfp4(torch.randn(N, K, device=DEV, generator=g) * 0.02)
        cases.append((M, N, K, b, b_sf, torch.empty(M, K, device=DEV), torch.empty(M, N, dtype=torch.bfloat16, device=DEV), torch.empty(M, N, device=DEV),
                      wb.MXFP4Linear(b, b_s)))

    def step(i, sync):
        outs = []
        for M, N, K, b, b_sf, x, c, acc, layer in cases:
            x.fill_(0.01 * (i + 1)).mul_(torch.arange(K, device=DEV) % 7 - 3.0)
            sync()
            q, s, sf = ops.quantize_mxfp4(x)
            sync()
            ops.scaled_gemm_packed(q, sf, b, b_sf, c)
            sync()
            acc.fill_(float(i))
            sync()
            ops.scaled_gemm_packed(q, ops.repack_scales(s), b, b_sf, acc, _lib.ACCUMULATE)
            sync()
            y = layer(x)
            sync()
            c.mul_(1.0)
            outs += [c.clone(), acc.clone(), y]
        return outs

    for _ in range(2):
        step(0, torch.cuda.synchronize)
    refs = [step(i, torch.cuda.synchronize) for i in range(12)]
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = [step(i, lambda: None) for i in range(12)]
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
    else:
        got = [step(i, lambda: None) for i in range(12)]
        torch.cuda.synchronize()
    for a, b in zip(got, refs):
        for u, v in zip(a, b):
            assert torch.equal(u, v)
    ops.check_device_status()


@pytest.mark.parametrize("kind,M,N,K", [("linear", 8, 640, 512), ("fp4", 16, 1024, 512), ("fp4", 256, 512, 4096), ("fp8", 16, 1024, 512), ("mixed", 16, 1024, 512)])
def test_a_capture_takes_the_memory_of_the_eager_call_before_it(kind, M, N, K, monkeypatch):
    """A layer or kernel object called on S, then on T, then again on S, and captured: the graph holds the workspace and the scratch of S,
    although the last call on S was recognised in native code. (At 256 rows the split-K workspace, which eager calls only ask for.)"""
    monkeypatch.setattr(ops, "_pool", ops.WorkspacePool())
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(M, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) * 0.02).to(DEV)
    if kind == "linear":
        layer = wb.MXFP4Linear.from_float(w)
        call, pool = (lambda: layer(x)), ops._pool
    else:
        if kind == "fp4":
            t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
            args = [*ops.quantize_mxfp4(x)[:2], *ops.quantize_mxfp4(w)[:2]]
        else:
            t, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4, "f8e4m3fn", wb.bf16,
                                                      weight_format="f4e2m1fn" if kind == "mixed" else None)
            options = wb.WaveCompileOptions(subs=subs)
            args = [*ops.quantize_mxfp8(x, torch.float8_e4m3fn)[:2], *(ops.quantize_mxfp4(w) if kind == "mixed" else ops.quantize_mxfp8(w, torch.float8_e4m3fn))[:2]]
        gemm = wb.wave_compile(wb.set_default_run_config(options), t)
        c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        call, pool = (lambda: (gemm(*args, c), c)[1]), gemm._workspaces if kind == "fp4" else ops._pool
    S, T, C = (torch.cuda.Stream(DEV) for _ in range(3))
    torch.cuda.synchronize()
    for st in (S, S, T, T, S):
        with torch.cuda.stream(st):
            ref = call().clone()
        torch.cuda.synchronize()
    captured = []
    get = ops.WorkspacePool.get
    monkeypatch.setattr(ops.WorkspacePool, "get", lambda *a: (captured.append(get(*a)), captured[-1])[1])
    if kind != "linear":
        scratch = gemm._a_scale_buffer
        monkeypatch.setattr(gemm, "_a_scale_buffer", lambda *a: (captured.append(scratch(*a)), captured[-1])[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=C):
        out = call()
    of_s = {pool._by_key[0, S.cuda_stream, "skinny" if M <= 128 else "splitk"].data_ptr()}
    if kind != "linear":
        of_s.add(gemm._a_scale_buf[0, S.cuda_stream][-1].data_ptr())
    assert {t.data_ptr() for t in captured} == of_s
    graph.replay()
    torch.cuda.synchronize()
    if M <= 128:  # (above, a captured call cuts K where an eager one does not)
        assert torch.equal(out, ref)
    ops.check_device_status()


@pytest.mark.parametrize("N,K", [(14336, 512), (4096, 1024), (28672, 256)])
def test_first_decode_calls_of_a_linear_layer_on_two_streams(N, K):
    """The first decode call of a layer stands behind queued work of its stream, the second one runs on another stream at once: both read
    packings that were complete before. Bits of a layer that is alone."""
    g = torch.Generator().manual_seed(N)
    w, x = (torch.randn(N, K, generator=g) * 0.02).to(DEV), torch.randn(8, K, generator=g).to(DEV)
    ref = wb.MXFP4Linear.from_float(w)(x)
    layer = wb.MXFP4Linear.from_float(w)
    blocks = [torch.full((ops.packed_scale_bytes(148 * 128, K),), 255, dtype=torch.uint8, device=DEV) for _ in range(4)]
    S, T = torch.cuda.Stream(DEV), torch.cuda.Stream(DEV)
    torch.cuda.synchronize()
    del blocks
    outs = []
    with torch.cuda.stream(S):
        torch.cuda._sleep(20_000_000)  # ~10 ms
        outs.append(layer(x))
    with torch.cuda.stream(T):
        outs += [layer(x), layer(x)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, ref) for y in outs)
    ops.check_device_status()


def test_linear_layer_packs_its_scales_for_every_decode_batch_and_anew_from_a_state_dict():
    from types import SimpleNamespace
    for N in (8, 130, 1000, 4096, 4097, 5803, 11008, 14336, 17800, 18900, 18944, 19072, 20480, 20483, 28672, 37888):
        for K in (32, 1024, 2080, 4096, 5376, 8192, 14336, 28672):
            for dtype in (torch.bfloat16, torch.float32):
                heights = {ops.decode_tile_rows_for(M, N, K, DEV, c_aligned=M == 1 or N * dtype.itemsize % 16 == 0) for M in range(1, 129)} - {128}
                layer = SimpleNamespace(out_features=N, in_features=K, output_dtype=dtype, weight_scales=torch.empty(0, device=DEV))
                assert len(heights) <= 1 and wb.MXFP4Linear._low_rows(layer) == min(heights, default=128)
    g = torch.Generator().manual_seed(4)
    one, two = (wb.MXFP4Linear.from_float((torch.randn(4096, 512, generator=g) * 0.02).to(DEV)) for _ in range(2))
    xs = [torch.randn(m, 512, generator=g).to(DEV) for m in (4, 300)]
    refs = [two(x) for x in xs]
    assert two._packed_low is not None and not torch.equal(one(xs[0]), refs[0])
    one.load_state_dict(two.state_dict())
    assert all(torch.equal(one(x), r) for x, r in zip(xs, refs))


def _two_stream_problem(n, M=8, N=2048, K=1024):
    """A kernel object, `n` weights (operands behind c), and the outputs of fresh kernel objects."""
    t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    compiled = lambda: wb.wave_compile(wb.set_default_run_config(options), t)  # noqa: E731
    probs = [[x.to(DEV) for x in random_problem(M, N, K, seed=60 + i)] for i in range(n)]
    refs = [torch.empty(M, N, dtype=torch.bfloat16, device=DEV) for _ in probs]
    for p, c in zip(probs, refs):
        compiled()(*p, c)
    blocks = [torch.full((ops.packed_scale_bytes(148 * 128, K),), 255, dtype=torch.uint8, device=DEV) for _ in range(8)]
    torch.cuda.synchronize()
    del blocks  # what is allocated next holds no scales
    return compiled(), probs, refs


def test_weight_scales_packed_on_one_stream_are_waited_for_on_another():
    """Both streams know the call. A weight's first call stands behind queued work of S; calls with that weight on T come at once, one of them while S's
    call is already one that native code recognises."""
    gemm, probs, refs = _two_stream_problem(3)
    S, T = torch.cuda.Stream(DEV), torch.cuda.Stream(DEV)
    outs = []

    def run(i, stream):
        with torch.cuda.stream(stream):
            c = torch.full_like(refs[i], float("nan"))
            gemm(*probs[i], c)
        outs.append((c, refs[i]))

    for stream in (S, T):
        run(0, stream)
        torch.cuda.synchronize()
    for i in (1, 2):
        with torch.cuda.stream(S):
            torch.cuda._sleep(20_000_000)  # ~10 ms
        for stream in (S, T, T) if i == 1 else (S, S, T, S, T):
            run(i, stream)
        torch.cuda.synchronize()
    for i in (1, 2):
        for _ in range(2):
            run(i, T)
    torch.cuda.synchronize()
    assert all(torch.equal(c, ref) for c, ref in outs)
    ops.check_device_status()


def test_packed_weight_scales_outlive_calls_of_another_stream():
    """A packing is dropped while a call of another stream that reads it is still queued: the memory goes to nobody on the stream it was made on."""
    gemm, probs, refs = _two_stream_problem(1)
    S, T = torch.cuda.Stream(DEV), torch.cuda.Stream(DEV)
    for stream in (S, T, T):
        with torch.cuda.stream(stream):
            gemm(*probs[0], torch.empty_like(refs[0]))
        torch.cuda.synchronize()
    outs = [torch.empty_like(refs[0]) for _ in range(2)]
    torch.cuda.synchronize()
    with torch.cuda.stream(T):
        torch.cuda._sleep(20_000_000)
        for c in outs:
            gemm(*probs[0], c)
    sizes = {p.data.numel() for _, p in gemm._weight_scales._entries.values()}
    gemm.drop_cached_weights()
    with torch.cuda.stream(S):
        blocks = [torch.full((n,), 255, dtype=torch.uint8, device=DEV) for n in sizes for _ in range(8)]
    torch.cuda.synchronize()
    assert len(blocks) and all(torch.equal(c, refs[0]) for c in outs)


def test_a_capture_while_weight_scales_are_being_packed():
    """Captured while the packing of its weight is still queued on another stream: the graph waits for nothing outside itself, so it packs
    the scales itself. Once the packing is complete, a capture takes it."""
    gemm, probs, refs = _two_stream_problem(2)
    S, C = torch.cuda.Stream(DEV), torch.cuda.Stream(DEV)
    with torch.cuda.stream(S):
        gemm(*probs[0], torch.empty_like(refs[0]))
    torch.cuda.synchronize()
    packings = []
    for complete in (False, True):
        with torch.cuda.stream(S):
            if not complete:
                torch.cuda._sleep(200_000_000)  # ~0.1 s
                gemm(*probs[1], torch.empty_like(refs[1]))
                behind = torch.cuda.Event()
                behind.record()
        before, c = gemm._weight_scales.packings, torch.full_like(refs[1], float("nan"))
        C.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(C):
            graph.capture_begin()
            gemm(*probs[1], c)
            graph.capture_end()
            packings.append(gemm._weight_scales.packings - before)
            if complete:
                graph.replay()
            else:
                pending = not behind.query()  # (otherwise this machine took its time, and nothing was pending any more)
        torch.cuda.synchronize()
        if not complete:  # (its scratch is that of the call on S)
            graph.replay()
            torch.cuda.synchronize()
        assert torch.equal(c, refs[1])
    assert packings == [1, 0] or not pending
    ops.check_device_status()


@pytest.mark.parametrize("rows", [4, 300])
def test_linear_refuses_codes_that_its_scales_were_not_packed_for(rows):
    """weight_codes replaced by a matrix of another size is refused as before any call was recognised in native code, and nothing is launched; nor is
    anything launched there on scales that are shorter than the matrix asks for."""
    N, K = 1024, 512
    g = torch.Generator().manual_seed(2)
    layer = wb.MXFP4Linear.from_float((torch.randn(N, K, generator=g) * 0.02).to(DEV))
    x = torch.randn(rows, K, generator=g).to(DEV)
    ref, codes = layer(x), layer.weight_codes
    for n, k in ((2 * N, K), (N // 2, K), (N + 8, K), (N, 2 * K)):
        layer.weight_codes = torch.zeros(n, k // 2, dtype=torch.uint8, device=DEV)
        with pytest.raises((ValueError, RuntimeError)):  # (another K: x does not fit)
            layer(x)
        if k == K:
            with pytest.raises(ValueError, match="do not agree"):
                layer(x)
    layer.weight_codes = codes
    packed, low = layer._packed, layer._packed_low
    native = lambda p, q, r=N, c=codes: _lib.fast().linear(x, c, (r, K, p, q, low.tile_rows), layer.output_dtype, ops._pool.fast)  # noqa: E731
    assert torch.equal(native(packed.data, low.data), ref)
    assert native(packed.data[:-512], low.data[:-512]) is None
    assert native(packed.data, low.data, N + 8) is None
    assert native(packed.data, low.data, N, codes.view(torch.int32).repeat(1, 4)) is None
    with pytest.raises(TypeError):
        _lib.fast().linear(x, codes, layer._native_scales, layer.output_dtype, [])
    assert torch.equal(layer(x), ref)
    ops.check_device_status()


def test_a_repeated_call_follows_weight_scales_that_were_given_another_view():
    """`scale.data = view` keeps the tensor, its address and its version. The packing belongs to the sizes and strides it was made with, also where
    the new ones are of a form that another weight's calls have made known."""
    M, N, K = 8, 512, 1024
    a, a_s, b, wide = (t.to(DEV) for t in random_problem(M, 2 * N, K, seed=5))
    b = b[:N].contiguous()
    t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    compiled = lambda: wb.wave_compile(wb.set_default_run_config(options), t)  # noqa: E731
    gemm, views = compiled(), (wide[:N], wide[::2])
    other, scale = wide.clone()[::2], torch.empty(0, dtype=torch.uint8, device=DEV)
    for s in (other, other, *views, *views):
        if s is not other:
            scale.data = s
            s = scale
        for _ in range(2):
            c, ref = (torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
            gemm(a, a_s, b, s, c)
            compiled()(a, a_s, b, s.clone(), ref)
            assert torch.equal(c, ref)
    ops.check_device_status()


@pytest.mark.parametrize("tiled", [False, True])
def test_weight_scales_packed_two_launches_ahead_of_an_overlapping_gemm(tiled):
    """The same chain with the scales of w packed by the repack entries: that kernel lets nothing start before it has ended, so the second
    GEMM, which may read them before its wait, finds them written. The first GEMM leaves most SMs free."""
    N, K, M = 16384, 8192, 16
    g = torch.Generator(device=DEV).manual_seed(6)
    lib, w = _lib.load(), torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device=DEV)
    scales = [torch.randint(110 + 12 * i, 115 + 12 * i, (N, K // 32), dtype=torch.uint8, generator=g, device=DEV) for i in range(2)]
    h = ops.decode_tile_rows_for(M, N, K) if tiled else 128
    assert tiled == (h != 128)
    pk = ops.repack_scales(scales[0], tile_rows=h)
    a, _, a_sf = ops.quantize_mxfp4(torch.randn(M, K, generator=g, device=DEV))
    q1, _, sf1 = ops.quantize_mxfp4(torch.randn(1024, K, generator=g, device=DEV))
    c1 = torch.empty(M, 1024, dtype=torch.bfloat16, device=DEV)
    refs = []
    for s in scales:
        ops.repack_scales(s, out=pk.data, tile_rows=h)
        torch.cuda.synchronize()
        refs.append(torch.empty(M, N, dtype=torch.bfloat16, device=DEV))
        ops.scaled_gemm_packed(a, a_sf, w, pk, refs[-1])
    outs = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(12)]
    for i, c in enumerate(outs):  # no synchronisation in between
        ops.repack_scales(scales[i & 1], out=pk.data, tile_rows=h)
        ops.scaled_gemm_packed(a, a_sf, q1, sf1, c1, _lib.OVERLAP_PREVIOUS)
        ops.scaled_gemm_packed(a, a_sf, w, pk, c, _lib.OVERLAP_PREVIOUS)
    torch.cuda.synchronize()
    for i, c in enumerate(outs):
        assert torch.equal(c.view(torch.int16), refs[i & 1].view(torch.int16))
    ops.check_device_status()


@pytest.mark.parametrize("kind,M", [("fp4", 64), ("fp4", 300), ("strided", 64), ("broadcast", 64), ("fp8", 64), ("mixed", 64)])
def test_threads_share_a_kernel_object_and_a_stream(kind, M):
    """Two threads call one kernel object on one stream, at sizes whose activation scales are packed into the object's scratch ahead of the GEMM: each
    call's two launches stay together. The scales of the threads are powers of two apart, so that the other one's would show."""
    import sys
    import threading
    N, K, calls = 1024, 2048, 400
    g = torch.Generator().manual_seed(M)
    bits = 8 if kind in ("fp8", "mixed") else 4
    if bits == 8:
        t, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4, "f8e4m3fn", wb.bf16,
                                                  weight_format="f4e2m1fn" if kind == "mixed" else None)
        options = wb.WaveCompileOptions(subs=subs)
    elif kind == "broadcast":
        t, subs = wb.get_broadcasted_scale_gemm_mxfp4((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4)
        options = wb.WaveCompileOptions(subs=subs)
    else:
        t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(wb.set_default_run_config(options), t)

    def operand(rows, bits):
        x = torch.randint(0, 256, (rows, K * bits // 8), dtype=torch.uint8, generator=g)
        return (x if bits == 4 else (x & 0xBF).view(torch.float8_e4m3fn)).to(DEV)

    a = operand(M, bits)
    if kind == "strided":
        a = torch.cat([a, a], 1)[:, :K // 2]
    b, b_s = operand(N, 8 if kind == "fp8" else 4), torch.randint(124, 131, (N, K // 32), dtype=torch.uint8, generator=g).to(DEV)
    scales = [torch.randint(110 + 20 * i, 115 + 20 * i, (M,) if kind == "broadcast" else (M, K // 32), dtype=torch.uint8, generator=g).to(DEV) for i in range(2)]
    dtype = t.output_dtype.torch_dtype
    outs = [[torch.empty(M, N, dtype=dtype, device=DEV) for _ in range(8)] for _ in scales]
    refs = [torch.empty(M, N, dtype=dtype, device=DEV) for _ in scales]
    for s, c in zip(scales, refs):
        gemm(a, s, b, b_s, c)
        torch.cuda.synchronize()
    wrong, start = [0, 0], threading.Barrier(2)

    def work(i):
        start.wait()
        for n in range(calls):
            gemm(a, scales[i], b, b_s, outs[i][n % 8])
            if n % 8 == 7:
                wrong[i] += sum(int(not torch.equal(c, refs[i])) for c in outs[i])

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
    finally:
        sys.setswitchinterval(interval)
    assert wrong == [0, 0]
    ops.check_device_status()


def test_a_workspace_that_is_not_aligned_is_no_obstacle_where_none_is_used():
    """Fewer 128-row tiles than SMs, one tile per SM: the whole-tile kernel, or with a workspace it cannot use the tile kernel that ran there before."""
    M, N, K = 16, 18800, 512
    a, a_s, b, b_s = random_problem(M, N, K, seed=7)
    ad, bd, a_sf, b_sf = a.to(DEV), b.to(DEV), ops.repack_scales(a_s.to(DEV)), ops.repack_scales(b_s.to(DEV))
    lib, ref = _lib.load(), orc.scaled_gemm(a, a_s, b, b_s)
    assert ops.decode_tile_rows_for(M, N, K) == 128
    n = int(lib.wb200_mxfp4_gemm_workspace_bytes(M, N, K))
    ws = torch.zeros(n + 16, dtype=torch.uint8, device=DEV)
    for shift in (0, 8):
        c = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        _lib.check(lib.wb200_mxfp4_gemm(M, N, K, ad.data_ptr(), a_sf.data.data_ptr(), bd.data_ptr(), b_sf.data.data_ptr(), c.data_ptr(), _lib.WB200_BF16, N,
                                        ws.data_ptr() + shift, n, 0, torch.cuda.current_stream().cuda_stream))
        check(c, a, a_s, b, b_s, ref=ref)
    ops.check_device_status()


def test_calls_in_inference_mode_are_recognised():
    """Tensors made in inference mode (every output of a layer there) take the native call as others do, with the bits of the ordinary ones. Weight scales
    made there have no version counter and are refused as before."""
    g = torch.Generator().manual_seed(8)
    layers = [wb.MXFP4Linear.from_float((torch.randn(512, 512, generator=g) * 0.05).to(DEV)) for _ in range(3)]
    x = torch.randn(8, 512, generator=g).to(torch.bfloat16).to(DEV)
    ref = layers[2](layers[1](layers[0](x)))
    M, N, K = 8, 640, 416
    t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    gemm = wb.wave_compile(wb.set_default_run_config(options), t)
    args = [v.to(DEV) for v in random_problem(M, N, K, seed=1)]
    c_ref = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    gemm(*args, c_ref)
    with torch.inference_mode(), pytest.MonkeyPatch.context() as mp:
        layers[0](x), gemm(*args, torch.empty_like(c_ref))
        mp.setattr(wb.MXFP4Linear, "_forward_checked", lambda *a: pytest.fail("left to the Python code"))
        y = layers[2](layers[1](layers[0](x)))
        assert y.is_inference() and torch.equal(y, ref)
        made = [v.clone() for v in args]
        for operands in ([*made[:3], args[3]], [*made[:3], args[3]]):
            c = torch.full_like(c_ref, float("nan"))
            assert c.is_inference() and gemm._fast.call(*operands, c, options.decode_tiled_weight_scales, options.kernel_path) == 0
            assert torch.equal(c, c_ref)
        with pytest.raises(RuntimeError):
            gemm(*made, c)
    ops.check_device_status()


def test_one_kernel_object_over_many_weights(monkeypatch):
    """More layers than one object's tables held, each at a decode and a prefill size: packed once per size, recognised from the second walk on, given back when
    their weights are gone. Where a packing has to go, it is not one that native calls have just read."""
    N, K, n = 512, 256, 100
    t, options = wb.get_tagged_mxfp4_gemm((8, N, K), output_dtype=wb.bf16)
    options.dynamic_symbols = ["M"]
    gemm = wb.wave_compile(wb.set_default_run_config(options), t)
    weights = [[v.to(DEV) for v in random_problem(8, N, K, seed=i)[2:]] for i in range(n)]
    acts = [[v.to(DEV) for v in random_problem(m, N, K, seed=m)[:2]] for m in (8, 200)]
    heights = {ops.decode_tile_rows_for(8, N, K), 128}
    assert len(heights) == 2

    def walk():
        outs = []
        for b, b_s in weights:
            for a, a_s in acts:
                outs.append(torch.empty(a.shape[0], N, dtype=torch.bfloat16, device=DEV))
                gemm(a, a_s, b, b_s, outs[-1])
        return outs

    first, packed = walk(), gemm._weight_scales.packings
    assert packed == 2 * n
    with monkeypatch.context() as mp:
        mp.setattr(gemm, "_launch", lambda *a: pytest.fail("left to the Python code"))
        again = walk()
    assert all(torch.equal(x, y) for x, y in zip(first, again))
    check(first[0], acts[0][0].cpu(), acts[0][1].cpu(), *(v.cpu() for v in weights[0]))
    keep = weights[:2]
    del weights[:]
    weights += keep
    weights.append([v.clone() for v in keep[0]])
    walk()
    assert gemm._weight_scales.packings == 2 * n + 2 and len(gemm._weight_scales._entries) == 6
    gemm.drop_cached_weights()
    gemm._weight_scales.capacity = 2
    a, a_s = acts[0]
    c = torch.empty(8, N, dtype=torch.bfloat16, device=DEV)
    for i in (0, 1, 0, 0, 2):  # weight 0 is used through native calls only when room is made for weight 2
        gemm(a, a_s, *weights[i], c)
    owners = [owner() for owner, _ in gemm._weight_scales._entries.values()]
    assert [any(o is weights[i][1] for o in owners) for i in range(3)] == [True, False, True]
    ops.check_device_status()


def test_calls_without_the_host_module(monkeypatch):
    """Where the host module cannot be used every call takes the Python code, captured ones included, with the same bits."""
    from wave_b200.graphs import GraphedScaledGemm
    M, N, K = 16, 1024, 512
    t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    args = [v.to(DEV) for v in random_problem(M, N, K, seed=1)]
    layer, x = wb.MXFP4Linear(*args[2:]), torch.randn(M, K, device=DEV)
    c_ref, ref = torch.empty(M, N, dtype=torch.bfloat16, device=DEV), layer(x)
    wb.wave_compile(options, t)(*args, c_ref)
    monkeypatch.setattr(_lib, "_fast", False)
    monkeypatch.setattr(ops, "_pool", ops.WorkspacePool())
    gemm, c = wb.wave_compile(options, t), torch.empty_like(c_ref)
    for run in (lambda: gemm(*args, c), lambda: gemm(*args, c), GraphedScaledGemm(gemm, *args, c).replay):
        c.fill_(float("nan"))
        run()
        assert torch.equal(c, c_ref)
    assert torch.equal(layer(x), ref) and gemm._fast is None
    ops.check_device_status()


@pytest.mark.parametrize("where", ["handle", "function"])
def test_calls_through_a_library_that_was_replaced_are_seen(where, monkeypatch):
    """A caller that puts an object in the place of the library, or a function in the place of one of its functions, sees every call of the linear layer and of the
    templates, also of forms that native code knows; and none of them once it has taken that back."""
    M, N, K = 16, 1024, 512
    t, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=wb.bf16)
    t8, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), wb.ScaledMMAType.F32_16x16x128_F8F6F4, "f8e4m3fn", wb.bf16)
    gemm, gemm8 = wb.wave_compile(options, t), wb.wave_compile(wb.WaveCompileOptions(subs=subs), t8)
    args = [v.to(DEV) for v in random_problem(M, N, K, seed=1)]
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    args8 = [*ops.quantize_mxfp8(x, torch.float8_e4m3fn)[:2], *ops.quantize_mxfp8(w, torch.float8_e4m3fn)[:2]]
    layer, c = wb.MXFP4Linear(*args[2:]), torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    lib, seen = _lib.load(), []
    entries = ["wb200_mxfp4_gemm_repack_a", "wb200_mxfp8_gemm_repack_a", "wb200_mxfp4_gemm_quantize_a"]

    def calls():
        gemm(*args, c), gemm8(*args8, c), layer(x)

    def spy(name, fn):
        return lambda *a: (seen.append(name), fn(*a))[1]

    class Watched:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            return spy(name, fn) if name in entries else fn

    for _ in range(2):
        calls()
    with monkeypatch.context() as mp:
        if where == "handle":
            for obj in (gemm, gemm8):
                mp.setattr(obj, "_lib", Watched())
            mp.setattr(_lib, "load", lambda: gemm._lib)
        else:
            for name in entries:
                mp.setattr(lib, name, spy(name, getattr(lib, name)))
        for _ in range(2):
            calls()
        assert seen == 2 * entries
    calls()
    assert len(seen) == 6
    ops.check_device_status()


@pytest.mark.parametrize("rows", [4, 300])
def test_a_captured_linear_call_follows_a_state_dict(rows):
    """The graph holds the addresses of codes and packings: both stay where they are when a state dict is loaded, and a replay reads what it brought."""
    g = torch.Generator().manual_seed(rows)
    one, two = (wb.MXFP4Linear.from_float((torch.randn(4096, 512, generator=g) * 0.02).to(DEV)) for _ in range(2))
    x = torch.randn(rows, 512, generator=g).to(DEV)
    one(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = one(x)
    at = one._packed.data.data_ptr(), one._packed_low.data.data_ptr()
    one.load_state_dict(two.state_dict())
    assert at == (one._packed.data.data_ptr(), one._packed_low.data.data_ptr())
    graph.replay()
    assert torch.equal(y, two(x)) and torch.equal(one(x), two(x))
    ops.check_device_status()
