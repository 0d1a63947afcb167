"""GPU tests of the dense contraction alone (myea_b200_gemm_nt) against a float64 product: the kernel that the size chooses
(FMA tiles, tensor-core tiles from fp32), and operand panels forced by bits 8..16 of `engine` - single tiles, ragged edges in
all three dimensions (TMA zero fill, guarded epilogue), K tails that are not a multiple of a stage, accumulate mode, long K,
rows of different magnitude - and the FP32 FMA engine."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from myea_b200 import capi

pytestmark = pytest.mark.gpu


TILE_SINGLE, TILE_PAIR, TILE_WIDE, TILE_WIDE_WHOLE = 128 << 8, 2 << 8, 3 << 8, 4 << 8   # forced tile shapes (engine bits 8..16)
A_TRANSPOSED, B_TRANSPOSED = 1 << 17, 1 << 18                                            # operand handed over as [K][rows]


def _gemm(M, N, K, engine=0, accumulate=0, seed=0, positive=False, return_out=False):
    lib = capi.load()
    rng = np.random.default_rng(seed)
    gen = (lambda s: rng.uniform(0, 1, s)) if positive else rng.standard_normal
    A, B = gen((M, K)).astype(np.float32), gen((N, K)).astype(np.float32)
    C0 = rng.standard_normal((M, N)).astype(np.float32) if accumulate else np.zeros((M, N), np.float32)
    out = C0.copy()
    ms = C.c_float(0)
    Ain = np.ascontiguousarray(A.T) if engine & A_TRANSPOSED else A
    Bin = np.ascontiguousarray(B.T) if engine & B_TRANSPOSED else B
    rc = lib.myea_b200_gemm_nt(0, engine, M, N, K, Ain.ctypes.data, Bin.ctypes.data, out.ctypes.data, accumulate, C.byref(ms), 0)
    assert rc == 0
    want = A.astype(np.float64) @ B.astype(np.float64).T + (C0 if accumulate else 0)
    err = float(np.abs(out - want).max() / np.abs(want).max())
    return (err, out) if return_out else err


SHAPES = [(128, 128, 32), (128, 256, 64), (1, 1, 1), (5, 3, 7), (100, 10, 256), (129, 130, 33), (300, 520, 100), (256, 64, 128), (512, 512, 512),
          (127, 1000, 2048)]


@pytest.mark.parametrize("shape", SHAPES)
def test_tcgen05_matches_float64(shape):
    """as the size chooses: (300, 520, 100), (512, 512, 512) and (127, 1000, 2048) run on tensor-core tiles, the others on FMA tiles"""
    assert _gemm(*shape) < 2e-5


@pytest.mark.parametrize("shape", SHAPES + [(257, 129, 65), (255, 385, 129), (1, 300, 191), (513, 1, 64)])
def test_operand_panels_match_float64(shape):
    assert _gemm(*shape, engine=TILE_WIDE) < 2e-5
    assert _gemm(*shape, engine=TILE_WIDE, accumulate=1) < 2e-5


@pytest.mark.parametrize("shape", [(64, 64, 16), (5, 3, 7), (300, 520, 100)])
def test_fma_engine_matches_float64(shape):
    assert _gemm(*shape, engine=1) < 2e-5


def test_accumulate_into_c():
    assert _gemm(256, 384, 512, accumulate=1) < 2e-5


def test_long_k_stays_accurate():
    # the multi-accumulator layout keeps a 16384-long sum within 3e-5 even for all-positive data (worst case for the
    # tensor core's truncating accumulate); zero-mean data is an order of magnitude better
    assert _gemm(256, 256, 16384) < 3e-5
    assert _gemm(256, 256, 16384, positive=True) < 1e-4


def test_forced_256_wide_tile():
    assert _gemm(256, 512, 1024, engine=(256 << 8)) < 5e-5


@pytest.mark.parametrize("tile", [TILE_SINGLE, TILE_PAIR, TILE_WIDE, TILE_WIDE_WHOLE])
@pytest.mark.parametrize("shape", [(256, 256, 64), (300, 520, 100), (1000, 777, 333), (129, 130, 33)])
def test_every_tile_shape(tile, shape):
    assert _gemm(*shape, engine=tile) < 2e-5


@pytest.mark.parametrize("shape", [(300, 520, 4096), (1024, 512, 2048), (2048, 1024, 1024), (640, 896, 8200), (2048, 2048, 8192)])
def test_tiles_split_along_k_are_exact_and_repeatable(shape):
    """fewer tiles than SM pairs: the 256 x 256 kernel cuts the K chunks of the tiles into equal runs (stream-K); the
    partial sums are added in a fixed order, so two runs agree bit for bit"""
    e1, o1 = _gemm(*shape, engine=TILE_WIDE, return_out=True)
    e2, o2 = _gemm(*shape, engine=TILE_WIDE, return_out=True)
    e3 = _gemm(*shape, engine=TILE_WIDE_WHOLE)
    assert e1 < 2e-5 and e3 < 2e-5
    assert np.array_equal(o1, o2)
    assert _gemm(*shape, engine=TILE_WIDE, accumulate=1) < 2e-5


@pytest.mark.parametrize("flags", [A_TRANSPOSED, B_TRANSPOSED, A_TRANSPOSED | B_TRANSPOSED])
@pytest.mark.parametrize("shape", [(256, 256, 64), (512, 768, 1000), (1000, 3000, 777), (130, 129, 136)])
def test_operands_read_through_their_columns(flags, shape):
    """MN-major operands of the 256 x 256 kernel: the source is [K][rows] and is not transposed on the way"""
    assert _gemm(*shape, engine=TILE_WIDE | flags) < 2e-5
    assert _gemm(*shape, engine=1 | TILE_WIDE | flags) < 2e-5   # the FP32 FMA engine on the same panels


@pytest.mark.parametrize("tile", [TILE_SINGLE, TILE_PAIR, TILE_WIDE])
@pytest.mark.parametrize("shape", [(256, 256, 64), (300, 520, 100), (1024, 512, 2048)])
def test_fused_activation_derivative_epilogue(tile, shape):
    """bit 19: C = (A B^T) .* relu'(C_in) - the epilogue of the error-propagation product, staged through shared memory"""
    M, N, K = shape
    lib = capi.load()
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    pre = rng.standard_normal((M, N)).astype(np.float32)
    out = pre.copy()
    rc = lib.myea_b200_gemm_nt(0, tile | (1 << 19), M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, 0, None, 0)
    assert rc == 0
    want = (A.astype(np.float64) @ B.astype(np.float64).T) * (pre >= 0)
    assert float(np.abs(out - want).max() / np.abs(want).max()) < 2e-5


def test_invalid_arguments():
    lib = capi.load()
    assert lib.myea_b200_gemm_nt(0, 0, 0, 4, 4, None, None, None, 0, None, 0) == -1


def test_operand_panels_of_many_million_rows():
    """more row blocks than the second dimension of a grid holds (65535 of 128 rows)"""
    lib = capi.load()
    M, N, K = 65536 * 128 + 1, 5, 16
    rng = np.random.default_rng(0)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = np.zeros((M, N), np.float32)
    assert lib.myea_b200_gemm_nt(0, 0, M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, 0, None, 0) == 0
    for rows in (slice(0, 1000), slice(M // 2, M // 2 + 1000), slice(M - 1000, M)):
        assert rel_err(out[rows], A[rows].astype(np.float64) @ B.astype(np.float64).T) < 5e-6


# Every row of C depends on its own row of A and every column on its own row of B: rows of very different magnitude and
# values that are not finite must leave their neighbours alone.  Bound: both operands keep 22 bits of a row's largest elements, an
# element below 2^-17 of them 2^-39 of the largest; 4096 products of random sign leave less than 2e-6 of |a| |b| per entry.
READINGS = [0, A_TRANSPOSED, B_TRANSPOSED, A_TRANSPOSED | B_TRANSPOSED]


def _product(A, B, engine):
    lib = capi.load()
    out = np.zeros((A.shape[0], B.shape[0]), np.float32)
    Ain = np.ascontiguousarray(A.T) if engine & A_TRANSPOSED else A
    Bin = np.ascontiguousarray(B.T) if engine & B_TRANSPOSED else B
    assert lib.myea_b200_gemm_nt(0, engine | TILE_WIDE, A.shape[0], B.shape[0], A.shape[1], Ain.ctypes.data, Bin.ctypes.data, out.ctypes.data, 0, None, 0) == 0
    return out


@pytest.mark.parametrize("engine", READINGS)
@pytest.mark.parametrize("M,N,K", [(300, 520, 700), (257, 100, 4096)])
@pytest.mark.parametrize("spread", [20, 45])
def test_rows_of_different_magnitude(M, N, K, engine, spread):
    rng = np.random.default_rng(M + K)
    A = (rng.standard_normal((M, K)) * 2.0 ** rng.uniform(-spread, spread, (M, 1))).astype(np.float32)
    B = (rng.standard_normal((N, K)) * 2.0 ** rng.uniform(-spread, spread, (N, 1))).astype(np.float32)
    A *= (2.0 ** rng.integers(-8, 9, K)).astype(np.float32)   # and of different columns: along K the other operand takes part in the sum
    A[7] = 0
    a, b = A.astype(np.float64), B.astype(np.float64)
    scale = np.linalg.norm(a, axis=1)[:, None] * np.linalg.norm(b, axis=1)[None, :]
    err = np.abs(_product(A, B, engine) - a @ b.T)
    assert not np.any(err[7]) and (err / np.maximum(scale, 1e-300)).max() < 2e-6


@pytest.mark.parametrize("engine", READINGS)
def test_values_that_are_not_finite_stay_in_their_row_and_column(engine):
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((300, 700)).astype(np.float32), rng.standard_normal((260, 700)).astype(np.float32)
    clean = A.astype(np.float64) @ B.astype(np.float64).T
    A[3, 77], A[140, 650], A[141, 5] = np.inf, np.nan, -np.inf
    B[9, 300], B[255, 699] = -np.inf, np.nan
    out = _product(A, B, engine)
    rows, cols = np.ones(300, bool), np.ones(260, bool)
    rows[[3, 140, 141]], cols[[9, 255]] = False, False
    assert rel_err(out[rows][:, cols], clean[rows][:, cols]) < 5e-6
    assert not np.isfinite(out[~rows]).any() and not np.isfinite(out[:, ~cols]).any()
