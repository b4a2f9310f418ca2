"""GPU parity tests of the tcgen05 GEMM behind nn::Linear and attention, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

from conftest import elementwise_excess, parity_record, relerr
from sptorch_b200.backend import BF16, EPI_GELU, EPI_SWIGLU, F32, MM_BF16, MM_F32, MM_TF32, bf16_bits_to_f32, f32_to_bf16_bits

pytestmark = pytest.mark.gpu


def _bf16(x):
    return bf16_bits_to_f32(f32_to_bf16_bits(x)).reshape(np.shape(x))


SHAPES = [(1, 8, 8), (128, 64, 64), (128, 64, 256), (129, 72, 257), (256, 768, 768), (512, 768, 3072), (300, 136, 200),
          (512, 3072, 768), (64, 4096, 512), (1000, 40, 50257 // 64)]


@pytest.mark.parametrize("M,K,N", SHAPES)
def test_linear_tf32_and_bf16_vs_oracle(backend, oracle, M, K, N):
    rng = np.random.default_rng(M + K + N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.01 * rng.standard_normal(N)).astype(np.float32)
    ref = oracle.linear(x, w, b, fast=2)
    assert relerr(backend.linear(x, w, b, mode=MM_TF32), ref) <= 2e-3          # north star: TF32 within 2e-3
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), ref) <= 2e-2          # north star: bf16 within 2e-2
    assert relerr(backend.linear(x, w, b, mode=MM_F32), ref) <= 5e-6           # CUDA-core f32 FMA
    # bf16 path against the oracle fed the same bf16-rounded operands: only the output rounding remains
    refb = oracle.linear(_bf16(x), _bf16(w), b, fast=2)
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), refb) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32), refb) <= 1e-5


@pytest.mark.parametrize("M,K,N", [(129, 768, 65), (512, 128, 384), (1000, 3072, 768), (1000, 72, 1160), (127, 100, 9472), (127, 100, 9473)])
def test_linear_narrow_tiles_where_they_all_run_at_once(backend, oracle, M, K, N):
    """64-column tiles: ragged last tiles of rows and columns, residual and bias, the largest N of 128 rows that takes them on 148 SMs and one
    more.  Same sums as every other tile width: one output rounding in bf16, 11-bit operands in TF32."""
    rng = np.random.default_rng(M + 3 * K + N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.01 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    assert relerr(backend.linear(x, w, b, residual=r, mode=MM_TF32), oracle.linear(x, w, b, fast=2) + r) <= 2e-3
    if K % 8 == 0:
        refb = oracle.linear(_bf16(x), _bf16(w), b, fast=2)
        assert relerr(backend.linear(x, w, b, mode=MM_BF16), refb) <= 2 ** -8 * 1.1
        assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16), oracle.unary("gelu", refb) + _bf16(r)) <= 2 ** -8 * 1.1


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("K,N", [(8, 1), (256, 7), (264, 1184), (768, 1185), (1024, 2369), (1032, 888), (1544, 1776), (2048, 1777), (2056, 592), (3072, 296), (3080, 148), (3080, 149), (3080, 297), (4096, 295), (4104, 296)])
def test_linear_of_a_row_or_a_few(backend, oracle, M, K, N):
    """A warp per group of weight rows: every number of vectors a lane holds and one element group more, outputs at the changes of the group size
    and at the last count that is resident at once, rows that divide a CTA's warps and rows that do not.  One output rounding in bf16."""
    rng = np.random.default_rng(M * 7 + K + N)
    x = _bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = _bf16((0.05 * rng.standard_normal((N, K))).astype(np.float32))
    b = (0.1 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    ref = oracle.linear(x, w, b, fast=2)
    assert relerr(backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32), ref) <= 1e-5
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), ref) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16), oracle.unary("gelu", ref) + _bf16(r)) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, None, alpha=0.5, mode=MM_BF16, out_dtype=F32), 0.5 * oracle.linear(x, w, None, fast=2)) <= 1e-5


@pytest.mark.parametrize("M,K,N", [(70, 8, 72), (300, 32, 200), (300, 40, 200), (130, 64, 136), (1000, 256, 768), (1000, 384, 768), (1000, 392, 520), (2100, 384, 768), (130, 776, 64),
                                   (5000, 72, 1032), (5000, 264, 1032)])
def test_linear_where_k_does_not_fill_the_ring(backend, oracle, M, K, N):
    """One to three stages, four, one k-block more than f32 outputs with a residual take four for, and launches with several tiles a CTA, which go
    around the ring.  TF32: a sum over K of products that are off by 2^-10 each; bf16: the output's rounding."""
    rng = np.random.default_rng(M + K + N)
    x, w = rng.standard_normal((M, K)).astype(np.float32), (K ** -0.5 * rng.standard_normal((N, K))).astype(np.float32)
    b, r = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    ref = oracle.linear(x, w, b, fast=2)
    assert relerr(backend.linear(x, w, b, residual=r, mode=MM_TF32), ref + r) <= 2e-3
    assert relerr(backend.linear(x, w, b, mode=MM_TF32), ref) <= 2e-3
    refb = oracle.linear(_bf16(x), _bf16(w), b, fast=2)
    assert relerr(backend.linear(x, w, b, residual=r, mode=MM_BF16), refb + _bf16(r)) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32), refb) <= 1e-5


@pytest.mark.parametrize("M,K,N", [(1000, 768, 3072), (4100, 136, 680), (4000, 64, 745), (254, 104, 14208), (254, 104, 14209)])
def test_linear_tiles_of_192_columns(backend, oracle, M, K, N):
    """192 columns where no narrower tiles all run at once: ragged last tiles of rows, columns and K, the largest N of 256 rows that takes them on
    148 SMs and one more (which goes back to 256), an output pitch that no tensor map describes.  The sums are those of CTA pairs on 256 columns,
    bit for bit."""
    rng = np.random.default_rng(M + 3 * K + N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.01 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    columns, paired = C.c_int(), C.c_int()
    outs = {}
    try:
        for pair in (1, 3):
            backend._check(backend.lib.sptorch_ext_set_gemm_pair(pair), "set_gemm_pair")
            backend._check(backend.lib.sptorch_ext_gemm_tile(M, N, K, MM_BF16, 0, C.byref(columns), C.byref(paired)), "gemm_tile")
            assert columns.value == (192 if pair == 3 and N != 14209 else 256)
            outs[pair] = [backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16), backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32),
                          backend.linear(x, w, b, residual=r, mode=MM_TF32)]
    finally:
        backend.lib.sptorch_ext_set_gemm_pair(3)
    for a, c in zip(outs[1], outs[3]):
        assert np.array_equal(a, c)
    assert relerr(outs[3][1], oracle.linear(_bf16(x), _bf16(w), b, fast=2)) <= 1e-5


@pytest.mark.parametrize("M,K,N,mode,columns,pair", [(8192, 2040, 384, MM_TF32, 192, 0), (8192, 2048, 384, MM_TF32, 256, 1), (8192, 2048, 384, MM_BF16, 192, 0), (4096, 3072, 768, MM_TF32, 256, 1),
                                                     (2040, 3072, 1536, MM_TF32, 192, 0)])
def test_long_tf32_products_of_many_rows_stay_on_pairs(backend, M, K, N, mode, columns, pair):
    """Where 192-column tiles all run at once but a long TF32 product is faster on pairs of CTAs."""
    c, p = C.c_int(), C.c_int()
    backend._check(backend.lib.sptorch_ext_gemm_tile(M, N, K, mode, 0, C.byref(c), C.byref(p)), "gemm_tile")
    assert (c.value, p.value) == (columns, pair)


@pytest.mark.parametrize("M", [4096, 16384])
@pytest.mark.parametrize("K,N", [(768, 768), (768, 3072), (3072, 768), (4096, 4096)])
def test_linear_sweep_shapes_vs_oracle(backend, oracle, M, K, N):
    """The standalone Linear sweep at its large row counts with the inputs it specifies (x ~ N(0,1), W ~ N(0,0.02), b ~ N(0,0.01),
    seeded per shape): every output element of the bf16 and the TF32 path against the oracle's f32 product (blocked, all host
    threads; no rows are left out)."""
    from sptorch_b200 import synth
    seed = 1000 * (M // 512) + K + N
    x = synth.normal(seed, M * K).reshape(M, K)
    w = synth.normal(seed + 1, N * K, std=0.02).reshape(N, K)
    b = synth.normal(seed + 2, N, std=0.01)
    ref = oracle.linear(x, w, b, fast=1)
    for mode, tol, name in ((MM_TF32, 2e-3, "tf32"), (MM_BF16, 2e-2, "bf16")):
        out = backend.linear(x, w, b, mode=mode)
        err = relerr(out, ref)
        outside, worst = elementwise_excess(out, ref, tol)
        parity_record(f"linear {M}x{K}->{N} {name}", relerr=err, elementwise_worst=worst)
        assert err <= tol, (name, err)
        assert worst <= 1.0, (name, outside, worst)


def test_linear_fused_epilogues(backend, oracle):
    rng = np.random.default_rng(1)
    M, K, N = 200, 128, 328
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.05 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.1 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    lin = oracle.linear(x, w, b, fast=2)
    ref = oracle.unary("gelu", lin) + r
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_TF32), ref) <= 2e-3
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_F32), ref) <= 5e-6
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16), ref) <= 2e-2
    assert relerr(backend.linear(x, w, None, alpha=0.5, mode=MM_TF32), 0.5 * oracle.linear(x, w, None, fast=2)) <= 2e-3


@pytest.mark.parametrize("M", [1, 3, 8, 16, 17, 33, 64])
@pytest.mark.parametrize("K,N", [(768, 768), (768, 2304), (3072, 768), (256, 50257 // 8), (96, 40), (64, 40), (56, 50257 // 8), (40, 10016)])
def test_linear_with_few_rows_vs_oracle(backend, oracle, M, K, N):
    """At most 64 input rows in bf16 (the projections of a decode step) run a weight-streaming kernel instead of 128-row tiles: up to 16 rows and
    3 M weights, and any rows where K is at most 64, the one with direct loads (one, two or four 16-row groups, one, two or four 8-row groups
    of weights per CTA), else the one with the weights as the wide tensor-core operand.  Against the oracle on the same bf16-rounded operands
    (only the output rounding remains), with the fused epilogues, and exactly on one-hot rows, where out[m, n] must be W[n, k_m]: every k
    position of an activation row has to meet the same k position of every weight row, ragged row and column counts included."""
    rng = np.random.default_rng(1000 * M + K + N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.01 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    refb = oracle.linear(_bf16(x), _bf16(w), b, fast=2)
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), refb) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), oracle.linear(x, w, b, fast=2)) <= 2e-2
    ref = oracle.unary("gelu", refb) + _bf16(r)
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16), ref) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, None, alpha=0.5, mode=MM_BF16), 0.5 * oracle.linear(_bf16(x), _bf16(w), None, fast=2)) <= 2 ** -8 * 1.1
    ks = rng.integers(0, K, M)
    onehot = np.zeros((M, K), np.float32)
    onehot[np.arange(M), ks] = 1.0
    wi = rng.integers(-64, 65, (N, K)).astype(np.float32)
    assert np.array_equal(backend.linear(onehot, wi, mode=MM_BF16), wi[:, ks].T)


@pytest.mark.parametrize("M,K,N", [(17, 72, 1), (17, 128, 129), (32, 200, 127), (33, 1000, 300), (64, 4104, 520), (64, 136, 33001), (3, 2048, 2056), (1, 5632, 2048),
                                   (16, 3000, 1500), (8, 768, 50257), (64, 2048, 3072), (48, 2056, 3072), (24, 768, 5632), (33, 768, 5632)])
def test_linear_with_the_weights_as_the_wide_operand(backend, oracle, M, K, N):
    """Row counts, ragged weight tiles and splits of K (one k-block per CTA, unequal parts, no split) of the streaming kernel on the tensor
    cores: bias, gate and residual, bf16 and f32 output (f32 sums of K products in another order than the oracle's: below sqrt(K) 2^-24 of
    the operands' scale, and bf16 outputs one rounding), rows whose pitch allows no vector stores."""
    rng = np.random.default_rng(7 * M + K + N)
    x = _bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = _bf16((0.02 * rng.standard_normal((N, K))).astype(np.float32))
    b = (0.01 * rng.standard_normal(N)).astype(np.float32)
    r = _bf16(rng.standard_normal((M, N)).astype(np.float32))
    ref = oracle.linear(x, w, b, fast=2)
    assert relerr(backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32), ref) <= 1e-5
    assert relerr(backend.linear(x, w, b, mode=MM_BF16), ref) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, residual=r, mode=MM_BF16), ref + r) <= 2 ** -8 * 1.1
    assert relerr(backend.linear(x, w, b, residual=r, epilogue=EPI_SWIGLU, mode=MM_BF16), r * ref / (1 + np.exp(-ref))) <= 2 ** -8 * 1.1


def test_linear_with_few_rows_on_tcgen05_tiles():
    """Row counts up to 64 take the weight-streaming kernel by default; SPTORCH_B200_FEW_ROWS=0 (read once per process, hence the
    child process) sends them through the 128-row tcgen05 tiles instead, which must agree with the oracle too."""
    import os, subprocess, sys, textwrap
    code = textwrap.dedent("""
        import numpy as np
        from sptorch_b200.backend import FfiBackend, MM_BF16, EPI_GELU, bf16_bits_to_f32, f32_to_bf16_bits
        from oracle import binding as oracle
        b = FfiBackend.load()
        r16 = lambda x: bf16_bits_to_f32(f32_to_bf16_bits(x)).reshape(np.shape(x))
        rel = lambda a, r: float(np.linalg.norm(a - r) / np.linalg.norm(r))
        for M, K, N in [(33, 768, 768), (64, 768, 2304), (64, 3072, 768), (48, 256, 6282)]:
            rng = np.random.default_rng(M + K + N)
            x = rng.standard_normal((M, K)).astype(np.float32)
            w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
            bias = (0.01 * rng.standard_normal(N)).astype(np.float32)
            res = rng.standard_normal((M, N)).astype(np.float32)
            ref = oracle.linear(r16(x), r16(w), bias, fast=2)
            assert rel(b.linear(x, w, bias, mode=MM_BF16), ref) <= 2 ** -8 * 1.1
            assert rel(b.linear(x, w, bias, residual=res, epilogue=EPI_GELU, mode=MM_BF16), oracle.unary("gelu", ref) + r16(res)) <= 2 ** -8 * 1.1
            ks = rng.integers(0, K, M)
            onehot = np.zeros((M, K), np.float32)
            onehot[np.arange(M), ks] = 1.0
            wi = rng.integers(-64, 65, (N, K)).astype(np.float32)
            assert np.array_equal(b.linear(onehot, wi, mode=MM_BF16), wi[:, ks].T)
        b.close()
        print("ok")
    """)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, SPTORCH_B200_FEW_ROWS="0", PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr


@pytest.mark.parametrize("width", [128, 256])
def test_linear_with_a_forced_tile_width(width):
    """SPTORCH_B200_GEMM_BN (read once per process, hence the child process): problems that would take narrower tiles by themselves, ragged in
    rows and columns, exact on integers and with the fused epilogues."""
    import os, subprocess, sys, textwrap
    code = textwrap.dedent("""
        import ctypes as C
        import numpy as np
        from sptorch_b200.backend import EPI_GELU, F32, FfiBackend, MM_BF16, MM_TF32
        from oracle import binding as oracle
        b = FfiBackend.load()
        rel = lambda a, r: float(np.abs(a - r).max() / np.abs(r).max())
        b._check(b.lib.sptorch_ext_set_gemm_pair(0), "set_gemm_pair")
        for M, K, N in [(129, 64, 129), (300, 72, 257), (70, 200, 600), (1000, 768, 1000)]:
            columns, pair = C.c_int(), C.c_int()
            for mode in (MM_TF32, MM_BF16):
                b._check(b.lib.sptorch_ext_gemm_tile(M, N, K, mode, 0, C.byref(columns), C.byref(pair)), "gemm_tile")
                assert (columns.value, pair.value) == (WIDTH, 0)
            rng = np.random.default_rng(M + K + N)
            xi, wi = rng.integers(-4, 5, (M, K)).astype(np.float32), rng.integers(-2, 3, (N, K)).astype(np.float32)
            assert np.array_equal(b.linear(xi, wi, mode=MM_BF16, out_dtype=F32), xi @ wi.T)
            assert np.array_equal(b.linear(xi, wi, mode=MM_TF32), xi @ wi.T)
            x, w = rng.standard_normal((M, K)).astype(np.float32), (0.05 * rng.standard_normal((N, K))).astype(np.float32)
            bias, r = (0.1 * rng.standard_normal(N)).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
            ref = oracle.unary("gelu", oracle.linear(x, w, bias, fast=2)) + r
            assert rel(b.linear(x, w, bias, residual=r, epilogue=EPI_GELU, mode=MM_TF32), ref) <= 2e-3
            assert rel(b.linear(x, w, bias, residual=r, epilogue=EPI_GELU, mode=MM_BF16), ref) <= 2e-2
        b.close()
        print("ok")
    """).replace("WIDTH", str(width))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, SPTORCH_B200_GEMM_BN=str(width), PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr


def test_linear_is_linear_at_full_size(backend):
    """Size-independent property at a shape of the standalone Linear sweep (M 4096, K 768, N 3072): f(x1 + x2) = f(x1) + f(x2) and
    integer-valued operands give exact integers."""
    rng = np.random.default_rng(2)
    M, K, N = 4096, 768, 3072
    x = rng.integers(-4, 5, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (N, K)).astype(np.float32)
    out = backend.linear(x, w, mode=MM_BF16, out_dtype=F32)
    ref = (x.astype(np.int32) @ w.astype(np.int32).T).astype(np.float32)
    assert np.array_equal(out, ref)                       # exact: every product and partial sum is a small integer
    assert np.array_equal(backend.linear(x, w, mode=MM_TF32), ref)


@pytest.mark.parametrize("M,K,N", [(1100, 512, 50304), (8320, 512, 50304), (300, 64, 1000), (4100, 64, 328)])
def test_tile_rasterisation_covers_every_tile_exactly_once(backend, M, K, N):
    """Integer-valued operands make every output exact, so a tile that is skipped, doubled or misplaced by the tile decode shows
    up as a wrong integer.  Shapes: a B operand above 48 MB (64-tile bands: one ragged band, then a full band plus a ragged
    one) and small operands (8-tile bands with ragged tails)."""
    rng = np.random.default_rng(M + N)
    x = rng.integers(-4, 5, (M, K)).astype(np.float32)
    w = rng.integers(-2, 3, (N, K)).astype(np.float32)
    ref = x @ w.T                                            # exact in f32: |sum| <= 8 * 512
    assert np.array_equal(backend.linear(x, w, mode=MM_BF16, out_dtype=F32), ref)
    assert np.array_equal(backend.linear(x, w, mode=MM_TF32), ref)


@pytest.mark.parametrize("M,K,N", [(129, 64, 129), (256, 64, 256), (640, 200, 328), (1000, 768, 1000), (2048, 3072, 768), (4100, 136, 50257 // 16)])
def test_pair_tiles_equal_single_cta_tiles(backend, oracle, M, K, N):
    """Wide problems run on CTA pairs (256 x 256 tiles, one MMA over two SMs).  Every output element is still the same
    k-ordered f32 accumulation, so the result must be bit-identical to the one-CTA kernel's, whatever the width of its tiles; both are
    checked against the oracle.  Asked for pairs, every shape takes them.  Shapes cover a second row half that is partly or wholly outside the matrix and ragged N."""
    rng = np.random.default_rng(M * 7 + N)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = (0.05 * rng.standard_normal((N, K))).astype(np.float32)
    b = (0.1 * rng.standard_normal(N)).astype(np.float32)
    r = rng.standard_normal((M, N)).astype(np.float32)
    ref = oracle.unary("gelu", oracle.linear(x, w, b, fast=2)) + r
    columns, paired = C.c_int(), C.c_int()
    try:
        outs = {}
        for pair in (1, 0, 3):
            backend._check(backend.lib.sptorch_ext_set_gemm_pair(pair), "set_gemm_pair")
            for mode in (MM_TF32, MM_BF16) if pair < 3 else ():
                backend._check(backend.lib.sptorch_ext_gemm_tile(M, N, K, mode, 0, C.byref(columns), C.byref(paired)), "gemm_tile")
                assert paired.value == pair and (columns.value == 256 or not pair)
            outs[pair] = [backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_TF32),
                          backend.linear(x, w, b, residual=r, epilogue=EPI_GELU, mode=MM_BF16),
                          backend.linear(x, w, b, mode=MM_BF16, out_dtype=F32)]
    finally:
        backend.lib.sptorch_ext_set_gemm_pair(3)           # the default: pairs where they measured faster
    for a, c, d in zip(outs[1], outs[0], outs[3]):
        assert np.array_equal(a, c) and np.array_equal(d, c)
    assert relerr(outs[1][0], ref) <= 2e-3
    assert relerr(outs[1][1], ref) <= 2e-2


@pytest.mark.parametrize("B,T,H,hd", [(2, 64, 4, 32), (1, 256, 2, 64), (2, 128, 2, 128), (1, 1024, 1, 64), (3, 8, 2, 32)])
def test_attention_vs_oracle(backend, oracle, B, T, H, hd):
    rng = np.random.default_rng(B * T + hd)
    d = H * hd
    q, k, v = (rng.standard_normal((B, T, d)).astype(np.float32) for _ in range(3))
    eye = np.eye(d, dtype=np.float32)
    # oracle: the reference's MHA with identity projections is exactly the attention core
    ref = np.stack([_mha_core(oracle, q[i], k[i], v[i], H) for i in range(B)])
    assert relerr(backend.attention_causal(q, k, v, H, dtype=F32), ref) <= 2e-3
    assert relerr(backend.attention_causal(q, k, v, H, dtype=BF16), ref) <= 2e-2
    del eye


def _mha_core(oracle, q, k, v, H):
    T, d = q.shape
    hd = d // H
    out = np.empty_like(q)
    for h in range(H):
        sl = slice(h * hd, (h + 1) * hd)
        s = oracle.matmul(q[:, sl], oracle.transpose(k[:, sl]), f64=True)[None]
        p = oracle.causal_softmax(s, 1.0 / np.sqrt(np.float32(hd)))[0]
        out[:, sl] = oracle.matmul(p, v[:, sl], f64=True)
    return out


@pytest.mark.parametrize("B,T,H,hd", [(1, 8, 1, 64), (2, 128, 3, 64), (1, 200, 2, 64), (2, 384, 2, 64), (1, 1024, 2, 64), (1, 136, 2, 128), (2, 512, 1, 128)])
def test_fused_attention_matches_materialised_and_oracle(backend, oracle, B, T, H, hd):
    """The fused kernel (scores never leave the SM) against the three-launch materialised form and the oracle,
    including sequence lengths that are not a multiple of the 128-row tile."""
    rng = np.random.default_rng(T + hd)
    d = H * hd
    q, k, v = (_bf16(rng.standard_normal((B, T, d)).astype(np.float32)) for _ in range(3))
    fused = backend.attention_causal(q, k, v, H, dtype=BF16)
    backend.lib.sptorch_ext_set_attention_mode(1)
    try:
        mat = backend.attention_causal(q, k, v, H, dtype=BF16)
    finally:
        backend.lib.sptorch_ext_set_attention_mode(0)
    ref = np.stack([_mha_core(oracle, q[i], k[i], v[i], H) for i in range(B)])
    assert relerr(fused, ref) <= 2e-2 and relerr(mat, ref) <= 2e-2
    assert relerr(fused, ref) <= 1.5 * 2 ** -8           # one bf16 rounding of P and of the output
    assert np.array_equal(fused[:, 0, :], v[:, 0, :])    # row 0 attends only to itself: output = V[0] exactly


@pytest.mark.parametrize("T,hd", [(8, 64), (128, 64), (136, 128), (248, 64), (256, 128), (264, 64), (1000, 64)])
def test_fused_attention_items_of_one_tile_equal_items_of_two(backend, oracle, T, hd):
    """Few enough sequences for every 128-row query tile to have an SM give each tile a work item of its own, more of them pair the tiles: the
    bits of a sequence alone are those it has among 150."""
    rng = np.random.default_rng(T + hd)
    H = 2
    q, k, v = (_bf16(rng.standard_normal((150, T, H * hd)).astype(np.float32)) for _ in range(3))
    many = np.asarray(backend.attention_causal(q, k, v, H, dtype=BF16))
    alone = np.asarray(backend.attention_causal(q[7:8], k[7:8], v[7:8], H, dtype=BF16))
    assert np.array_equal(alone[0], many[7])
    assert relerr(alone[0], _mha_core(oracle, q[7], k[7], v[7], H)) <= 1.5 * 2 ** -8


@pytest.mark.parametrize("B,T,H,hd", [(1, 4, 1, 4), (3, 28, 2, 32), (2, 32, 3, 36), (2, 64, 2, 64), (1, 68, 2, 68), (2, 100, 5, 20), (2, 128, 3, 128), (40, 36, 7, 64)])
def test_short_f32_attention_in_one_launch(backend, oracle, B, T, H, hd):
    """f32 sequences of up to 128 tokens: one key, ragged query and key tiles, head sizes at and past the edges of its three instantiations.  All
    f32 multiply-adds: a score of scale 3 sharp over 128 products is off by sqrt(128) 2^-24 of that, 2e-6 sharp, and so is its weight; the oracle's
    f32 softmax as much again (the three-launch form rounds its operands to eleven bits, 2e-3).  A sequence alone besides."""
    rng = np.random.default_rng(T + hd)
    q, k, v = (rng.standard_normal((B, T, H * hd)).astype(np.float32) for _ in range(3))
    for sharp in (1.0, 20.0):
        out = np.asarray(backend.attention_causal(sharp * q, k, v, H, dtype=F32))
        ref = np.stack([_mha_core(oracle, sharp * q[i], k[i], v[i], H) for i in range(B)])
        assert relerr(out, ref) <= 4e-6 * sharp
        assert np.array_equal(out[:, 0], v[:, 0])            # row 0 attends only to itself
    assert np.array_equal(np.asarray(backend.attention_causal(sharp * q[:1], k[:1], v[:1], H, dtype=F32))[0], out[0])


@pytest.mark.parametrize("T,hd", [(36, 32), (100, 64), (128, 128)])
def test_short_f32_attention_with_values_that_are_not_finite(backend, T, hd):
    """Queries, keys and values side by side in one buffer (the model's pitch), the bits of separate ones.  A key or a query that is NaN reaches the rows that
    see it and no other; a score of minus infinity has no weight; an infinite value is its column's result."""
    rng = np.random.default_rng(T)
    H, d = 2, 2 * hd
    qkv = rng.standard_normal((2, T, 3 * d)).astype(np.float32)
    ws, out = backend.alloc(backend.lib.sptorch_ext_attention_workspace(2, T, H, hd, F32), 1), backend.alloc(2 * T * d)
    def attend(x):
        b = backend.upload(x)
        at = b.handle
        backend._check(backend.lib.sptorch_ext_attention_causal(at, at + 4 * d, at + 8 * d, out.handle, ws.handle, 2, T, H, hd, 3 * d, F32), "attention")
        y = out.to_host().reshape(2, T, d)
        b.free()
        return y
    clean = attend(qkv)
    assert np.array_equal(clean, np.asarray(backend.attention_causal(*(np.ascontiguousarray(qkv[..., i * d:(i + 1) * d]) for i in range(3)), H, dtype=F32)))
    at = T // 2 + 1
    x = qkv.copy()
    x[0, at, d + 3] = np.nan                                                  # a key of the first head
    y = attend(x)
    assert np.isnan(y[0, at:, :hd]).all() and np.array_equal(y[0, :at], clean[0, :at]) and np.array_equal(y[0, :, hd:], clean[0, :, hd:]) and np.array_equal(y[1], clean[1])
    x = qkv.copy()
    x[1, at, hd] = np.nan                                                     # a query of the second
    y = attend(x)
    assert np.isnan(y[1, at, hd:]).all()
    y[1, at, hd:] = clean[1, at, hd:]
    assert np.array_equal(y, clean)
    x = qkv.copy()
    x[0, :, 0], x[0, at, d] = np.abs(x[0, :, 0]) + 0.1, -np.inf               # a key that every query of the first head scores minus infinity
    y = attend(x)
    x[0, at, d], x[0, at, 2 * d:2 * d + hd] = -1e30, 0.0
    assert np.array_equal(y[0, :, :hd], attend(x)[0, :, :hd]) and np.isfinite(y[0, :at]).all()
    x = qkv.copy()
    x[0, 0, 2 * d + 5] = np.inf                                               # a value that every row of the first head sees
    y = attend(x)
    assert np.isposinf(y[0, :, 5]).all()
    y[0, :, 5] = clean[0, :, 5]
    assert np.array_equal(y, clean)
    ws.free(), out.free()


@pytest.mark.parametrize("B,T,H,hd", [(64, 128, 12, 64), (64, 36, 12, 32), (3, 256, 2, 64)])
def test_f32_attention_over_one_of_its_inputs(backend, B, T, H, hd):
    """f32 attention may put its output where the queries, the keys or the values are: nothing is written before everyone has read it.  More blocks than run
    at once.  Over q the one launch serves as it is; the others' products are TF32."""
    rng = np.random.default_rng(T)
    n = B * T * H * hd
    host = [rng.standard_normal(n).astype(np.float32) for _ in range(3)]
    ref = np.asarray(backend.attention_causal(*(x.reshape(B, T, H * hd) for x in host), H, dtype=F32)).reshape(-1)
    ws = backend.alloc(backend.lib.sptorch_ext_attention_workspace(B, T, H, hd, F32), 1)
    try:
        for over in range(3):
            bufs = [backend.upload(x) for x in host]
            backend._check(backend.lib.sptorch_ext_attention_causal(*(x.handle for x in bufs), bufs[over].handle, ws.handle, B, T, H, hd, H * hd, F32), "attention")
            assert relerr(bufs[over].to_host(), ref) <= (1e-30 if over == 0 else 2e-3), "qkv"[over]
            for x in bufs:
                x.free()
    finally:
        ws.free()


@pytest.mark.parametrize("T,hd", [(256, 64), (384, 128), (200, 64)])
def test_fused_attention_with_steeply_rising_scores(backend, oracle, T, hd):
    """Scores that grow by far more than 2^8 from one 32-key chunk to the next (key j = 8 (j // 4) u, query = u): the running row maximum
    of the fused kernel moves at every chunk, so everything accumulated under the old maximum -- the row sum, the output in TMEM and
    the part of P already written for the current tile -- is rescaled each time.  The softmax is then concentrated on the last
    few visible keys; the result must still match the oracle within one bf16 rounding of P and of the output."""
    rng = np.random.default_rng(T + hd)
    H = 2
    u = np.where(rng.random(hd) < 0.5, -0.125, 0.125).astype(np.float32)
    q = np.tile(u, (1, T, H)).astype(np.float32)
    k = np.concatenate([(8.0 * (j // 4)) * np.tile(u, H)[None, :] for j in range(T)])[None].astype(np.float32)
    v = _bf16(rng.standard_normal((1, T, H * hd)).astype(np.float32))
    assert np.array_equal(_bf16(k), k)                     # the keys are exact in bf16
    fused = backend.attention_causal(q, k, v, H, dtype=BF16)
    ref = _mha_core(oracle, q[0], k[0], v[0], H)[None]
    assert relerr(fused, ref) <= 1.5 * 2 ** -8
    # and the other way round: falling scores never move the maximum after the first chunk
    k2 = k[:, ::-1].copy()
    fused2 = backend.attention_causal(q, k2, v, H, dtype=BF16)
    ref2 = _mha_core(oracle, q[0], k2[0], v[0], H)[None]
    assert relerr(fused2, ref2) <= 1.5 * 2 ** -8
@pytest.mark.parametrize("T", [264, 320, 384, 640, 896])
def test_fused_attention_when_the_last_query_tile_is_alone(backend, oracle, T):
    """T = 256 n + 1 .. 128: the last work item has one query tile, whose scores run two key tiles ahead of P V.  The first warp's rows are
    slow (their maximum moves at every chunk), the other warps' rows are not, so the fast warps ask for the last product long before it --
    or the ones before it -- is done; none of them may read the output early."""
    rng = np.random.default_rng(T)
    B, H, hd = 2, 8, 64
    u = np.where(rng.random(hd) < 0.5, -0.125, 0.125).astype(np.float32)
    q = _bf16(0.02 * rng.standard_normal((B, T, H * hd)).astype(np.float32))
    last = (T - 1) // 128 * 128
    q[:, last:last + 32] = np.tile(u, H)
    k = np.concatenate([(8.0 * (j // 4)) * np.tile(u, H)[None, :] for j in range(T)])[None].repeat(B, 0).astype(np.float32)
    k = _bf16(k)
    v = _bf16(rng.standard_normal((B, T, H * hd)).astype(np.float32))
    ref = np.stack([_mha_core(oracle, q[i], k[i], v[i], H) for i in range(B)])
    for _ in range(5):
        assert relerr(backend.attention_causal(q, k, v, H, dtype=BF16), ref) <= 2e-2


@pytest.mark.parametrize("T", [40, 300, 600, 830])
def test_fused_attention_items_with_and_without_a_second_query_tile(backend, oracle, T):
    """T = 256 n + 1 .. 128 on more (sequence, head, tile pair) items than SMs: a CTA goes from an item with one query tile to items with
    two, and the warps of the absent tile must neither start on the next item's scores early nor free its accumulator twice."""
    rng = np.random.default_rng(T)
    B, H, hd = 32, 12, 64
    q, k, v = (_bf16(rng.standard_normal((B, T, H * hd)).astype(np.float32)) for _ in range(3))
    ref = np.stack([_mha_core(oracle, q[i], k[i], v[i], H) for i in (0, B - 1)])
    first = None
    for _ in range(4):
        out = np.asarray(backend.attention_causal(q, k, v, H, dtype=BF16))
        assert relerr(out[[0, B - 1]], ref) <= 2e-2 and np.isfinite(out).all()
        first = out if first is None else first
        assert np.array_equal(out, first)
