"""GPU tests of the paths small and middle networks take, at the edges of their tiles: contractions straight from fp32
operands (16 x 16 and 32 x 32 FMA tiles; 128 x 64 tensor-core tiles, 32 of K per stage, K cut over 1, 2, 4 or 8 CTAs), the one-launch
normalization of short batches (8 columns per block, 4 to 32 rows per thread), the LSTM walks (resident weights: groups of 1
to many CTAs, clusters, chunks of exchange data; which pass takes which), widths of one, and the updates and products that leave or read
operand panels - against float64 products and the numpy restatement."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from myea_b200 import capi, workloads
from myea_b200.net import Net
from oracle import myea_oracle

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _plan(M, N, K, columns=0):
    """(rows of a tile, CTAs that share one): 16 and 32 with FMAs, 128 on the tensor cores straight from fp32, 256 from operand panels"""
    tile, ctas = C.c_int(), C.c_int()
    assert capi.load().myea_b200_contraction_plan(C.c_uint64(M), C.c_uint64(N), C.c_uint64(K), columns >> 17, C.byref(tile), C.byref(ctas)) == 0
    return tile.value, ctas.value


# (the size chooses: (64, 640, 2048) runs on tensor-core tiles, (257, 10, 1000) and (5, 4, 4099) on FMA tiles of 32 x 32 over clusters, the others on
# FMA tiles of 16 x 16)
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 64, 7), (3, 65, 31), (127, 63, 32), (128, 64, 33), (129, 65, 64), (130, 130, 257), (257, 10, 1000), (64, 640, 2048),
                                   (5, 4, 4099)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_contraction_from_fp32_operands(M, N, K, accumulate):
    lib = capi.load()
    rng = np.random.default_rng(M * 7 + N * 3 + K)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = rng.standard_normal((M, N), dtype=np.float32)
    want = A.astype(np.float64) @ B.astype(np.float64).T + (out if accumulate else 0)
    assert lib.myea_b200_gemm_nt(0, 0, M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, accumulate, None, 0) == 0
    assert rel_err(out, want) < 5e-6


# edges of the chunks of K (128, 124 where rows start off 16-byte boundaries) and of the 16 x 16 tiles, through rows and columns
@pytest.mark.parametrize("K", [1, 3, 8, 123, 124, 125, 128, 129, 249, 256, 257, 333, 513])
@pytest.mark.parametrize("M,N", [(1, 1), (17, 33), (203, 333), (128, 256)])
@pytest.mark.parametrize("engine", [0, 1 << 17, 1 << 18, 3 << 17])
def test_contraction_from_fp32_operands_over_k(M, N, K, engine):
    lib = capi.load()
    assert _plan(M, N, K, engine) == (16, 1)
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = np.zeros((M, N), np.float32)
    a, b = np.ascontiguousarray(A.T) if engine & (1 << 17) else A, np.ascontiguousarray(B.T) if engine & (1 << 18) else B
    assert lib.myea_b200_gemm_nt(0, engine, M, N, K, a.ctypes.data, b.ctypes.data, out.ctypes.data, 0, None, 0) == 0
    assert rel_err(out, A.astype(np.float64) @ B.astype(np.float64).T) < 5e-6


def _step(wl, seed=5, kinks=0.0):
    """one training step and one inference pass on the GPU and on the restatement; kinks: bound in the 2-norm of the derivatives, and of the
    outputs behind the update that they make, where single elements may take the other branch of an activation's derivative"""
    gpu, cpu = Net(wl.desc, wl.opt), myea_oracle.OracleNet(wl.desc, wl.opt)
    X, Y = wl.batch(seed)
    for net in (gpu, cpu):
        wl.materialize(net)
        net.reset_loss(); net.forward(X); net.compute_error(Y); net.backward(); net.update_derivative_weight()
    out = [(gpu.outputs(len(wl.layers) - 1), cpu.outputs(len(wl.layers) - 1)), (gpu.get(capi.BUF_DERIVATIVES), cpu.get(capi.BUF_DERIVATIVES))]
    for net in (gpu, cpu):
        net.update_parameter()
        net.forward(X, training=False)
    out += [(gpu.get(capi.BUF_PARAMETERS), cpu.get(capi.BUF_PARAMETERS)), (gpu.outputs(len(wl.layers) - 1), cpu.outputs(len(wl.layers) - 1))]
    if gpu.n_norm:
        out += [(gpu.get(b), cpu.get(b)) for b in (capi.BUF_NORM_MEAN_AVERAGE, capi.BUF_NORM_VARIANCE_AVERAGE)]
    gpu.synchronize()
    gpu.close()
    if kinks:
        for got, want in (out.pop(3), out.pop(1)):
            assert np.linalg.norm(got - want) < kinks * np.linalg.norm(want)
    for got, want in out:
        assert rel_err(got, want) < TOL


def _mlp(widths, B, af, norm=capi.NORM_NONE, drop=capi.DROP_NONE):
    layers = [capi.fc(widths[0])] + [capi.fc(w, af, norm, drop, (0.7, 0, 0)) for w in widths[1:-1]] + [capi.fc(widths[-1], capi.AF_LINEAR)]
    return workloads.Workload("edges", capi.net(layers, B, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE, r_max=3.0, d_max=5.0),
                              capi.opt(capi.OPT_GD, gd_lr=0.01 / B, momentum=0.9), widths[0], widths[-1], False, layers)


@pytest.mark.parametrize("widths,B", [((3, 5, 2), 1), ((31, 33, 7), 31), ((32, 64, 64), 33), ((65, 63, 129, 4), 127), ((64, 128, 256, 8), 128), ((129, 130, 65), 129),
                                      ((300, 70, 71, 72, 73, 74, 75, 76, 77, 78, 79, 80, 81, 82), 65)])
@pytest.mark.parametrize("af", [capi.AF_TANH, capi.AF_SINE])
def test_plain_networks(widths, B, af):
    _step(_mlp(widths, B, af, drop=capi.DROP_BERNOULLI))


@pytest.mark.parametrize("B", [7, 31, 128, 129, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("norm", [capi.NORM_BN, capi.NORM_BRN])
def test_normalized_short_batches(B, norm):
    _step(_mlp((9, 37, 16, 3), B, capi.AF_SIGMOID, norm, capi.DROP_BERNOULLI_INVERTED))


# normalizations and activations that write operand panels: ragged blocks of 128 rows and columns, masked units
@pytest.mark.parametrize("widths,B", [((1000, 1048, 904, 130), 700), ((512, 1032, 1160, 64), 1025)])
@pytest.mark.parametrize("norm", [capi.NORM_NONE, capi.NORM_BN, capi.NORM_BRN])
def test_producers_of_operand_panels(widths, B, norm):
    _step(_mlp(widths, B, capi.AF_TANH, norm, capi.DROP_BERNOULLI_INVERTED))


# residual blocks whose products run on operand panels (from 600 Mi multiply-adds on): column sums of a normalization from the product
# before it, forward and backward, and panels of the next block's first layer from the ShakeDrop kernel; rows that are a multiple of 32 and
# not, and a width that is none, where the sums are taken in a pass of their own
@pytest.mark.parametrize("H,B", [(1024, 704), (1024, 700), (1000, 700)])
@pytest.mark.parametrize("norm,af", [(capi.NORM_BN, capi.AF_TANH), (capi.NORM_BRN, capi.AF_TANH), (capi.NORM_BN, capi.AF_ELU), (capi.NORM_BRN, capi.AF_SIGMOID)])
@pytest.mark.parametrize("depth", [2, 3])
def test_residual_blocks_on_operand_panels(H, B, norm, af, depth):
    """The derivative of ELU (as the reference has it) jumps from 0 to 1 at 0: pre-activations within rounding of it, about 2e-6 of
    B * H * 7 layers or 10 elements, may take either side, and each is sqrt(1 / (B * H)) of its layer's error: 4e-3 in the 2-norm."""
    assert H * H * B > 600 << 20
    layers = [capi.fc(40), capi.fc(H, af)]
    for _ in range(2):
        layers += [capi.residual(depth, capi.DROP_SHAKEDROP, (0.5, 0.0, 0.0)), capi.fc(H, af)] + [capi.fc(H, af, norm) for _ in range(depth - 1)]
    layers.append(capi.fc(30, capi.AF_LINEAR))
    _step(workloads.Workload("blocks on panels", capi.net(layers, B, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE, r_max=3.0, d_max=5.0),
                             capi.opt(capi.OPT_GD, gd_lr=0.01 / B, momentum=0.9), 40, 30, False, layers), kinks=1e-2 if af == capi.AF_ELU else 0.0)


def _walk(net, layer=1):
    """what the forward and the backward pass of an LSTM layer take: [walk, CTAs per group, cluster, groups, row passes, rows per thread, one cell
    per thread]; walk 0 launches, 1 tensor cores, 2 resident weights"""
    out = []
    for kind in (1, 2):
        w = (C.c_int * 7)()
        assert net.lib.myea_b200_lstm_walk(net.h, layer, kind, w) == 0
        out.append(list(w))
    return out


# The resident walk on clusters: one to three steps (the barriers' first phases), rows and cells that do not divide; whether the forward and the
# backward pass runs on one, in how many row passes, with how many rows per thread, and whether a thread keeps one row and cell
@pytest.mark.parametrize("H,T,B,bidirectional,zoneout,forward,backward", [
    (150, 1, 50, False, 0.0, (1, 1, 4, 1), (1, 1, 4, 1)), (150, 2, 50, False, 0.1, (1, 1, 4, 1), (1, 1, 4, 1)), (203, 3, 61, False, 0.0, (1, 1, 4, 1), (0, 1, 4, 1)),
    (129, 7, 30, True, 0.2, (1, 1, 4, 1), (1, 1, 4, 1)), (120, 4, 200, False, 0.1, (1, 1, 4, 1), (1, 1, 4, 1)), (160, 4, 128, True, 0.0, (1, 1, 4, 1), (1, 1, 8, 1)),
    (150, 5, 256, True, 0.0, (1, 2, 4, 0), (0, 1, 8, 0)), (205, 3, 256, True, 0.1, (1, 2, 4, 0), (0, 1, 8, 0)), (180, 4, 250, True, 0.2, (1, 2, 4, 0), (0, 1, 4, 0)),
    (142, 4, 256, True, 0.1, (0, 1, 4, 1), (1, 1, 8, 0)), (142, 1, 255, True, 0.0, (0, 1, 4, 1), (1, 1, 8, 0))])
def test_lstm_walk_on_clusters(H, T, B, bidirectional, zoneout, forward, backward):
    wl = _one_lstm(5, H, T, B, bidirectional, zoneout)
    net = Net(wl.desc, wl.opt)
    walks = _walk(net)
    net.close()
    assert [(w[0], w[2], w[4], w[5], w[6]) for w in walks] == [(2,) + forward, (2,) + backward]
    _step(wl)


def _one_lstm(n_in, H, T, B, bidirectional, zoneout):
    layers = [capi.fc(n_in), capi.lstm(H, bidirectional=bidirectional, dropout=capi.DROP_ZONEOUT if zoneout else capi.DROP_NONE, p=(zoneout, zoneout, 0.0)),
              capi.fc(H, capi.AF_LINEAR)]
    return workloads.Workload("lstm edges", capi.net(layers, B, T=T, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE),
                              capi.opt(capi.OPT_GD, gd_lr=0.01 / B, momentum=0.9), n_in, H, False, layers)


@pytest.mark.parametrize("n_in,H,T,B,bidirectional,zoneout", [
    (3, 5, 4, 3, False, 0.0), (7, 32, 3, 5, True, 0.3), (11, 37, 5, 50, False, 0.2), (16, 64, 1, 4, False, 0.0), (20, 107, 3, 9, False, 0.0), (20, 150, 4, 50, True, 0.1),
    (9, 313, 3, 33, False, 0.0), (12, 512, 3, 70, False, 0.1), (5, 601, 3, 7, True, 0.0), (8, 1100, 2, 3, False, 0.0), (5, 300, 4, 5, False, 0.1),
    (5, 90, 5, 256, True, 0.0)])
def test_lstm_with_resident_weights(n_in, H, T, B, bidirectional, zoneout):
    _step(_one_lstm(n_in, H, T, B, bidirectional, zoneout))


@pytest.mark.parametrize("widths,B", [((1000, 904, 1100, 130), 700), ((1004, 1000, 1096), 640)])   # multiples of 8 and not, ragged blocks of 128
@pytest.mark.parametrize("opt", [dict(t=capi.OPT_ADAM, eps=1.0), dict(t=capi.OPT_AMSGRAD, eps=1.0, weight_decay=1e-3), dict(t=capi.OPT_GD, gd_lr=1e-5, momentum=0.9, nesterov=True, clip=0.5)])
def test_update_writes_operand_panels(widths, B, opt):
    """updates that leave the next step's weight panels and unzeroed derivatives: accumulation over two batches, derivatives read
    back, an update without any, parameters replaced from the host, inference between the steps"""
    kw = dict(opt)
    layers = [capi.fc(widths[0])] + [capi.fc(w, capi.AF_TANH) for w in widths[1:-1]] + [capi.fc(widths[-1], capi.AF_LINEAR)]
    wl = workloads.Workload("panels", capi.net(layers, B, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE), capi.opt(kw.pop("t"), **kw), widths[0], widths[-1], False, layers)
    gpu, cpu = Net(wl.desc, wl.opt), myea_oracle.OracleNet(wl.desc, wl.opt)
    out = []
    for net in (gpu, cpu):
        wl.materialize(net)
        got = []
        if opt.get("weight_decay"):
            mask = np.ones(gpu.P, np.float32)
            mask[::3] = 0
            net.set(capi.BUF_MASK_REGULARIZED, mask)
        for batches in (1, 2, 0, 1):
            for k in range(batches):
                X, Y = wl.batch(7 + k)
                net.reset_loss(); net.forward(X); net.compute_error(Y); net.backward(); net.update_derivative_weight()
            got.append(net.get(capi.BUF_DERIVATIVES) if batches == 2 else None)
            net.update_parameter()
            got.append(net.get(capi.BUF_PARAMETERS))
        assert not np.any(net.get(capi.BUF_DERIVATIVES))
        net.forward(X, training=False)
        got.append(net.outputs(len(widths) - 1))
        net.set(capi.BUF_PARAMETERS, got[1])
        net.forward(X, training=False)
        got.append(net.outputs(len(widths) - 1))
        out.append([g for g in got if g is not None])
    gpu.synchronize()
    gpu.close()
    for got, want in zip(*out):
        assert rel_err(got, want) < TOL


@pytest.mark.parametrize("M,N,K,tile", [
    (1, 1, 1, 16), (31, 33, 3, 16), (32, 32, 4, 16), (33, 65, 255, 16), (64, 96, 256, 16), (65, 31, 257, 16), (128, 256, 280, 16), (100, 37, 360, 16), (96, 128, 281, 16),
    (90, 50, 361, 16), (384, 384, 1, 32), (290, 310, 64, 32), (33, 2300, 130, 32), (300, 300, 255, 32), (320, 320, 256, 32), (300, 300, 257, 32), (257, 450, 281, 32),
    (301, 303, 361, 32)])
@pytest.mark.parametrize("columns", [0, 1 << 18, 3 << 17])   # both operands by rows, B by columns, both by columns
def test_contraction_with_fmas(M, N, K, tile, columns):
    """the FMA tiles of 16 x 16 and, uncut, of 32 x 32 at the edges of their rows, columns and the 128 and 256 of K that they hold at a time"""
    lib = capi.load()
    assert _plan(M, N, K, columns) == (tile, 1)
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = rng.standard_normal((M, N), dtype=np.float32)
    want = A.astype(np.float64) @ B.astype(np.float64).T + out
    a, b = np.ascontiguousarray(A.T if columns & (1 << 17) else A), np.ascontiguousarray(B.T if columns & (1 << 18) else B)
    assert lib.myea_b200_gemm_nt(0, columns, M, N, K, a.ctypes.data, b.ctypes.data, out.ctypes.data, 1, None, 0) == 0
    assert rel_err(out, want) < 5e-6


@pytest.mark.parametrize("M,N,K", [(257, 640, 64), (300, 520, 7), (385, 449, 31), (1, 4800, 33), (129, 1250, 65), (4801, 1, 40), (415, 417, 1000), (513, 321, 32),
                                   (128, 1216, 4036)])
@pytest.mark.parametrize("columns", [0, 1 << 17, 1 << 18, 3 << 17])   # which operands are read through their columns
@pytest.mark.parametrize("accumulate", [0, 1])
def test_contraction_on_tensor_core_tiles_from_fp32(M, N, K, columns, accumulate):
    """more than 148 tiles of 32 x 32, which is where the 128 x 64 tensor-core tile takes over: edges of its rows, columns and the
    32 of K of a stage, pitches that are not 16-byte aligned, K cut over a cluster"""
    lib = capi.load()
    assert -(-M // 32) * -(-N // 32) > 148 and _plan(M, N, K, columns)[0] == 128
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = rng.standard_normal((M, N), dtype=np.float32)
    want = A.astype(np.float64) @ B.astype(np.float64).T + (out if accumulate else 0)
    a, b = np.ascontiguousarray(A.T if columns & (1 << 17) else A), np.ascontiguousarray(B.T if columns & (1 << 18) else B)
    assert lib.myea_b200_gemm_nt(0, columns, M, N, K, a.ctypes.data, b.ctypes.data, out.ctypes.data, accumulate, None, 0) == 0
    assert rel_err(out, want) < 5e-6


@pytest.mark.parametrize("M,N,K,plan", [
    (64, 1024, 1000, (32, 2)), (65, 600, 900, (32, 2)), (1, 1000, 1000, (32, 4)), (700, 12, 1301, (32, 4)), (256, 10, 1024, (32, 8)), (33, 7, 1025, (32, 8)),
    (40, 31, 4099, (32, 8)), (1, 1, 600, (16, 1)), (64, 512, 512, (16, 1)), (65, 129, 515, (16, 1))])
def test_contraction_with_fmas_over_a_cluster(M, N, K, plan):
    """few tiles and a long K: cut over 2, 4 and 8 CTAs, the last share shorter; or, where they are as fast, tiles of 16 x 16"""
    lib = capi.load()
    assert _plan(M, N, K) == plan
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
    out = rng.standard_normal((M, N), dtype=np.float32)
    want = A.astype(np.float64) @ B.astype(np.float64).T + out
    assert lib.myea_b200_gemm_nt(0, 0, M, N, K, A.ctypes.data, B.ctypes.data, out.ctypes.data, 1, None, 0) == 0
    assert rel_err(out, want) < 5e-6


@pytest.mark.parametrize("widths,B", [((20, 30, 10), 640), ((5, 33, 40, 3), 1027)])   # weight derivatives with a long K: bias sums over a cluster
def test_derivatives_over_long_batches(widths, B):
    _step(_mlp(widths, B, capi.AF_TANH))


@pytest.mark.parametrize("widths", [(1, 1), (5, 7, 1), (1, 6, 4), (3, 1, 2), (9, 1, 1, 1, 5), (1, 40, 70, 1)])   # layers of one unit beside wider ones, one input
@pytest.mark.parametrize("B,norm", [(1, capi.NORM_NONE), (65, capi.NORM_NONE), (65, capi.NORM_BN)])
def test_layers_of_one_unit(widths, B, norm):
    _step(_mlp(widths, B, capi.AF_TANH, norm))


@pytest.mark.parametrize("n_in,H,out", [(1, 8, 8), (1, 37, 40), (4, 1, 1), (4, 1, 6), (1, 1, 1)])   # univariate series, layers of one cell
@pytest.mark.parametrize("T,B", [(1, 4), (5, 1), (4, 9)])
@pytest.mark.parametrize("bidirectional", [False, True])
def test_lstm_of_one_input_or_one_cell(n_in, H, out, T, B, bidirectional):
    layers = [capi.fc(n_in), capi.lstm(H, bidirectional=bidirectional), capi.fc(out, capi.AF_LINEAR)]
    _step(workloads.Workload("narrow lstm", capi.net(layers, B, T=T, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE),
                             capi.opt(capi.OPT_GD, gd_lr=0.01 / B, momentum=0.9), n_in, out, False, layers))


@pytest.mark.parametrize("spread_of", ["samples", "features"])
def test_panels_of_a_step_with_units_of_different_magnitude(spread_of):
    """samples or features, and units, spread over 2^+-18 (the largest weight derivative is 2^120 then) on a network whose products
    read operand panels: outputs, errors, weight derivatives and the outputs behind an update, each against float64 at its own
    scale (|row| |column| of the operands)"""
    n_in, H, n_out, B = 1000, 1096, 904, 700
    rng = np.random.default_rng(11)
    spread = lambda *shape: 2.0 ** rng.uniform(-18, 18, shape)
    layers = [capi.fc(n_in), capi.fc(H, capi.AF_LINEAR), capi.fc(n_out, capi.AF_LINEAR)]
    desc, opt = capi.net(layers, B, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE), capi.opt(capi.OPT_GD, gd_lr=2.0 ** -60)
    X = (rng.standard_normal((1, B, n_in)) * (spread(B, 1) if spread_of == "samples" else spread(n_in))).astype(np.float32)
    W1 = (rng.standard_normal((H, n_in)) * spread(H, 1)).astype(np.float32)
    W2 = (rng.standard_normal((n_out, H)) * spread(n_out, 1)).astype(np.float32)
    gpu = Net(desc, opt)
    p = np.zeros(gpu.P, np.float32)
    at = [int(gpu.layer_index(l).first_connection_index) for l in (1, 2)]
    p[at[0]:at[0] + W1.size], p[at[1]:at[1] + W2.size] = W1.ravel(), W2.ravel()
    gpu.set(capi.BUF_PARAMETERS, p)
    gpu.forward(X); gpu.compute_error(np.zeros((1, B, n_out), np.float32)); gpu.backward(); gpu.update_derivative_weight()
    norm = lambda a, axis: np.linalg.norm(a, axis=axis)

    def check(got, a, b, bias=0.0):   # got = a b^T + bias, all in float64
        scale = norm(a, 1)[:, None] * norm(b, 1)[None, :] + np.abs(bias)
        assert (np.abs(got - a @ b.T - bias) / scale).max() < 5e-6

    # every product against float64 on the operands the GPU itself computed
    f64 = lambda a: np.asarray(a, np.float64)
    x, h, y, g = f64(X[0]), f64(gpu.outputs(1)).reshape(B, H), f64(gpu.outputs(2)).reshape(B, n_out), f64(gpu.get(capi.BUF_DERIVATIVES))
    check(h, x, f64(W1)); check(y, h, f64(W2))
    check(g[at[1]:at[1] + W2.size].reshape(n_out, H), y.T, h.T)
    d1 = f64(gpu.errors(1)).reshape(B, H)
    check(d1, y, f64(W2).T)
    check(g[at[0]:at[0] + W1.size].reshape(H, n_in), d1.T, x.T)
    gpu.update_parameter()
    q = gpu.get(capi.BUF_PARAMETERS)
    gpu.forward(X, training=False)
    bias = int(gpu.layer_index(1).first_bias_connection_index)
    check(f64(gpu.outputs(1)).reshape(B, H), x, f64(q[at[0]:at[0] + W1.size]).reshape(H, n_in), f64(q[bias:bias + H]))
    gpu.synchronize()
    gpu.close()


@pytest.mark.parametrize("bidirectional", [False, True])
def test_lstm_errors_of_samples_of_different_magnitude(bidirectional):
    """the tensor-core walk back through time: samples whose errors lie 2^36 apart, each against float64 at its own scale (fp32
    gates and three steps of products leave about 1e-6)"""
    H, B, T = (1024, 136, 4) if not bidirectional else (512, 300, 3)
    layers = [capi.fc(9), capi.lstm(H, bidirectional=bidirectional), capi.fc(H, capi.AF_LINEAR)]
    wl = workloads.Workload("samples", capi.net(layers, B, T=T, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE), capi.opt(capi.OPT_GD, gd_lr=1e-6), 9, H, False, layers)
    gpu, cpu = Net(wl.desc, wl.opt), myea_oracle.OracleNet(wl.desc, wl.opt, dtype=np.float64)
    X, Y = wl.batch(5)
    Y = (Y + 1.0) * (2.0 ** np.random.default_rng(1).uniform(0, 36, (1, B, 1))).astype(np.float32)
    for net in (gpu, cpu):
        wl.materialize(net)
        net.forward(X); net.compute_error(Y); net.backward()
    got, want = np.asarray(gpu.errors(1), np.float64), np.asarray(cpu.layers[1].dh, np.float64).reshape(T, B, -1)
    assert (np.linalg.norm(got - want, axis=2) / np.linalg.norm(want, axis=2)).max() < 1e-5
    gpu.synchronize()
    gpu.close()


@pytest.mark.parametrize("n_in,H,T,B,bidirectional,zoneout", [
    (8, 1024, 3, 16, False, 0.2), (8, 512, 3, 64, True, 0.1), (8, 1024, 2, 40, False, 0.0),   # resident forward and tensor-core backward, both tensor-core
    (8, 1001, 3, 32, False, 0.2), (8, 601, 3, 128, True, 0.0)])                                # the same against the walk by launches
def test_lstm_passes_on_different_walks(n_in, H, T, B, bidirectional, zoneout):
    """every pass of a layer takes the walk that is estimated to be the fastest; two steps and an inference pass with new weights"""
    layers = [capi.fc(n_in), capi.lstm(H, bidirectional=bidirectional, dropout=capi.DROP_ZONEOUT if zoneout else capi.DROP_NONE, p=(zoneout, zoneout, 0.0)),
              capi.fc(H, capi.AF_LINEAR)]
    wl = workloads.Workload("walks", capi.net(layers, B, T=T, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE),
                            capi.opt(capi.OPT_GD, gd_lr=0.01 / B, momentum=0.9), n_in, H, False, layers)
    gpu, cpu = Net(wl.desc, wl.opt), myea_oracle.OracleNet(wl.desc, wl.opt)
    X, Y = wl.batch(5)
    out = []
    for net in (gpu, cpu):
        wl.materialize(net)
        got = []
        for step in range(2):
            net.reset_loss(); net.forward(X); net.compute_error(Y); net.backward(); net.update_derivative_weight()
            got += [net.outputs(1), net.errors(1), net.get(capi.BUF_DERIVATIVES)]
            net.update_parameter()
            got.append(net.get(capi.BUF_PARAMETERS))
        net.forward(X, training=False)
        out.append(got + [net.outputs(1)])
    gpu.synchronize()
    gpu.close()
    for got, want in zip(*out):
        assert rel_err(got, want) < TOL


def test_reciprocal_of_the_lstm_cells_against_the_correctly_rounded_one():
    """every float of [1, 2^126) against CUDA's __frcp_rn"""
    lib = capi.load()
    one, end = 0x3F800000, 0x7E800000
    different, most = C.c_uint64(), C.c_uint32()
    assert lib.myea_b200_reciprocal_check(0, one, end - one, C.byref(different), C.byref(most)) == 0
    assert different.value == 0 and most.value == 0


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("H,B,bidirectional,walks,stalls", [   # walks: of the forward and the backward pass, whether on clusters
    (1024, 136, False, ([1, 0], [1, 0]), (2,)), (150, 50, False, ([2, 1], [2, 1]), (1, 2, 3)), (512, 16, False, ([2, 0], [2, 0]), (1, 2, 3)),
    (150, 256, True, ([2, 1], [2, 0]), (1, 3)), (142, 256, True, ([2, 0], [2, 1]), (1, 3))])   # two row passes; several cells per thread
def test_a_step_barrier_that_is_never_reached_ends_in_an_error_status(H, B, bidirectional, walks, stalls, backward):
    """a walk whose wait gives up (after half a millisecond here; the tensor-core walk's other waits after a second), in the first, a middle and
    the last step: every copy and product in flight is waited for, the status is an error, and the GPU goes on - a new handle
    computes what the first one did"""
    T = 4
    layers = [capi.fc(9), capi.lstm(H, bidirectional=bidirectional), capi.fc(H, capi.AF_LINEAR)]
    wl = workloads.Workload("stall", capi.net(layers, B, T=T, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE), capi.opt(capi.OPT_GD, gd_lr=1e-6), 9, H, False, layers)
    X, Y = wl.batch(5)
    out = []
    for stall in (0,) + stalls + (0,):
        net = Net(wl.desc, wl.opt)
        assert [w[:3:2] for w in _walk(net)] == list(walks)
        wl.materialize(net)
        if not backward:
            assert net.lib.myea_b200_lstm_stall(net.h, stall, C.c_uint64(1 << 20)) == 0
        net.forward(X)
        if backward:
            net.compute_error(Y)
            assert net.lib.myea_b200_lstm_stall(net.h, stall, C.c_uint64(1 << 20)) == 0
            net.backward()
        rc = net.lib.myea_b200_synchronize(net.h)
        assert rc == (0 if stall == 0 else -3), net.lib.myea_b200_last_error(net.h)
        if stall == 0:
            out.append(net.errors(1) if backward else net.outputs(1))
        net.close()
    assert np.array_equal(out[0], out[1])


def test_a_second_backward_pass_does_not_read_the_errors_of_the_first():
    """compute_error and backward twice on one forward pass, with other targets, on layers that read operand panels"""
    layers = [capi.fc(1000), capi.fc(904, capi.AF_TANH), capi.fc(1096, capi.AF_TANH), capi.fc(1000, capi.AF_LINEAR)]
    wl = workloads.Workload("twice", capi.net(layers, 700, loss=capi.LOSS_MSE, accuracy=capi.ACC_DISTANCE), capi.opt(capi.OPT_GD, gd_lr=1e-6), 1000, 1000, False, layers)
    X, Y = wl.batch(5)
    out = []
    for targets in ((Y,), (Y + 1.0, Y)):
        net = Net(wl.desc, wl.opt)
        wl.materialize(net)
        net.forward(X)
        for t in targets:
            net.compute_error(t.astype(np.float32)); net.backward()
        net.update_derivative_weight()
        out.append(net.get(capi.BUF_DERIVATIVES))
        net.close()
    assert np.array_equal(out[0], out[1])
