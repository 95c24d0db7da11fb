"""GPU parity of the tensor-core W4A16 contraction (tcgen05) against the CPU oracle and against the
fused GEMV: every row of the batched result must equal the single-token result within fp32
summation order (at most one fp16 ulp, on few outputs)."""
import numpy as np
import pytest
import torch

from test_gemv_gpu import _to_dev, _ulp_diff

pytestmark = pytest.mark.gpu


def _gemm(ops, cuda, p, s, z, M, K, X, zp_integral=True):
    ws = ops.Workspace()
    w = ops.W4Linear(_to_dev(p, cuda), _to_dev(s, cuda), _to_dev(z, cuda), M, K, zp_integral=zp_integral)
    R = X.shape[0]
    pad = 64
    ybuf = torch.full((R * M + 2 * pad,), -7.0, dtype=torch.float16, device=cuda)
    y = ybuf[pad:pad + R * M].view(R, M)
    ops.gemm_w4a16(w, ws, _to_dev(X, cuda), y)
    ws.check()
    out = ybuf.cpu().numpy()
    assert (out[:pad] == np.float16(-7.0)).all() and (out[pad + R * M:] == np.float16(-7.0)).all()
    return out[pad:pad + R * M].reshape(R, M), w, ws


def _check(got, y32, y16, what, differ=0.01):
    err = np.abs(got.astype(np.float32) - y32)
    tol = 2e-2 * np.abs(y32) + 2e-2 * np.abs(y32).mean()
    assert (err <= tol).all(), f"{what}: max err {err.max()}"
    ulps = _ulp_diff(got, y16)
    tiny = np.abs(got.astype(np.float32) - y16.astype(np.float32)) <= 1e-4 * np.abs(y32).mean()
    assert ((ulps <= 1) | tiny).all(), f"{what}: {ulps[~tiny].max()} ulp"
    assert (ulps > 0).mean() < differ, f"{what}: {(ulps > 0).mean():.4f} differ"


@pytest.mark.parametrize("M,K,R", [(128, 128, 16), (256, 256, 16), (512, 512, 5), (1536, 512, 64), (512, 1536, 33),
                                   (1152, 512, 16), (2176, 512, 100), (640, 384, 256), (256, 1024, 300)])
def test_gemm_matches_oracle_small(ops, orc, cuda, M, K, R):
    p, s, z = orc.gen_linear(40, M, K)
    X = orc.gen_normal_f16(40, orc.ACT, R * K).reshape(R, K)
    y32, y16 = orc.gemm_w4a16(p, s, z, M, K, X)
    got, _, _ = _gemm(ops, cuda, p, s, z, M, K, X)
    _check(got, y32, y16, f"{M}x{K} rows {R}")


def test_gemm_fractional_zero_points(ops, orc, cuda):
    M, K, R = 512, 512, 16
    p, s, _ = orc.gen_linear(41, M, K)
    z = orc.gen_normal_f16(41, 999, M // 128, 7.5, 1.3)
    X = orc.gen_normal_f16(41, orc.ACT, R * K).reshape(R, K)
    y32, y16 = orc.gemm_w4a16(p, s, z, M, K, X)
    got, _, _ = _gemm(ops, cuda, p, s, z, M, K, X, zp_integral=False)
    _check(got, y32, y16, "generic zero-point path")


@pytest.mark.parametrize("M,K", [(12288, 4096), (4096, 4096), (4096, 12288), (151936, 4096)])
@pytest.mark.parametrize("R", [16, 64, 256, 2048])
def test_gemm_sweep_rows_equal_gemv(ops, orc, cuda, M, K, R):
    """The batched-row sweep at full size: a sample of rows against the CPU oracle, and every
    sampled row against the fused GEMV on the GPU."""
    kind = orc.UNEMB if M == 151936 else orc.WQKV
    p, s, z = orc.gen_linear(42, M, K, kind=kind)
    X = orc.gen_normal_f16(42, orc.ACT, R * K).reshape(R, K)
    got, w, ws = _gemm(ops, cuda, p, s, z, M, K, X)
    rows = sorted(set([0, R // 2, R - 1]))
    y32, y16 = orc.gemm_w4a16(p, s, z, M, K, X[rows])
    # the tensor cores add the fp32 products of a K=16 step with their own internal alignment, so a few
    # per cent of the fp16 results land on the other side of a rounding boundary (never more than one ulp)
    _check(got[rows], y32, y16, f"{M}x{K} rows {R}", differ=0.05 if K <= 4096 else 0.08)
    y = torch.zeros(M, dtype=torch.float16, device=cuda)
    for r in rows:
        ops.gemv_w4a16(w, ws, ops.gemv_args(_to_dev(X[r], cuda), y=y))
        yv = y.cpu().numpy()
        d = _ulp_diff(got[r], yv)
        near = np.abs(got[r].astype(np.float32) - yv.astype(np.float32)) <= 1e-4 * np.abs(yv.astype(np.float32)).mean()
        # one-ulp differences only; their share grows with the number of accumulation steps (K)
        assert ((d <= 1) | near).all() and (d > 0).mean() < (0.05 if K <= 4096 else 0.08)
    ws.check()


@pytest.mark.parametrize("M,K,R,integral", [
    (384, 512, 130, True),     # an odd number of 128-output blocks: the last pair has one CTA without outputs; fewest K blocks
    (256, 640, 161, True),     # K blocks that are no multiple of the rings and of the unpack groups
    (640, 1152, 159, False), (2176, 896, 160, True), (896, 2176, 193, False),   # group depends on the input, K not a power of two
    (4096, 512, 257, True), (1664, 1536, 129, True),                           # one row past a row tile
    (19200, 4096, 160, False),   # more tiles than pairs of SMs: a whole wave, then a tile whose K is split
    (256, 8192, 144, True)])     # one tile: K split over many pairs
def test_gemm_pairs_edges(ops, orc, cuda, M, K, R, integral):
    p, s, z = orc.gen_linear(43, M, K)
    if not integral:
        z = orc.gen_normal_f16(43, 999, M // 128, 7.5, 1.3)
    X = orc.gen_normal_f16(43, orc.ACT, R * K).reshape(R, K)
    got, w, ws = _gemm(ops, cuda, p, s, z, M, K, X, zp_integral=integral)
    rows = sorted(set([0, 1, R // 2, R - 2, R - 1]))
    y32, y16 = orc.gemm_w4a16(p, s, z, M, K, X[rows])
    _check(got[rows], y32, y16, f"{M}x{K} rows {R}", differ=0.05 if K <= 4096 else 0.08)
    # a result that does not start on 16 bytes takes the one-CTA kernel
    off = torch.zeros(R * M + 8, dtype=torch.float16, device=cuda)
    y = off[2:2 + R * M].view(R, M)
    ops.gemm_w4a16(w, ws, _to_dev(X, cuda), y)
    ws.check()
    d = _ulp_diff(y.cpu().numpy(), got)
    near = np.abs(y.cpu().numpy().astype(np.float32) - got.astype(np.float32)) <= 1e-4 * np.abs(y32).mean()
    assert ((d <= 1) | near).all() and (d > 0).mean() < 0.08


@pytest.mark.parametrize("M,K,R", [(12288, 4096, 2048), (4096, 12288, 300)])
def test_gemm_pairs_repeat_bitwise(ops, orc, cuda, M, K, R):
    """Several waves of tiles, and single tiles with long sums, 60 launches each: an operand that one CTA of a pair reads before the
    other's writes have arrived would show as a difference between launches."""
    p, s, z = orc.gen_linear(46, M, K)
    ws = ops.Workspace()
    w = ops.W4Linear(_to_dev(p, cuda), _to_dev(s, cuda), _to_dev(z, cuda), M, K)
    x = _to_dev(orc.gen_normal_f16(46, orc.ACT, R * K).reshape(R, K), cuda)
    first = torch.zeros(R, M, dtype=torch.float16, device=cuda)
    ops.gemm_w4a16(w, ws, x, first)
    y = torch.zeros_like(first)
    for _ in range(60):
        ops.gemm_w4a16(w, ws, x, y)
        assert torch.equal(y, first)
    ws.check()


@pytest.mark.parametrize("M,K,R", [(19200, 4096, 64), (4096, 1024, 256)])
def test_gemm_pairs_sum_no_longer_than_one_cta(ops, orc, cuda, M, K, R):
    """The error of a result grows with the number of MMAs that one accumulator sums.  Share of results that are not the nearest fp16 of
    the 64-bit sum: the pairs' against the one-CTA kernel's (a result off 16 bytes), of some hundred each, so that twice the
    length (1.8 times the share) is ten standard deviations away from the bound."""
    p, s, z = orc.gen_linear(47, M, K)
    X = orc.gen_normal_f16(47, orc.ACT, R * K).reshape(R, K)
    rows = np.arange(0, R, R // 64 * 4 if M < 10000 else R // 16)
    _, want = orc.gemm_w4a16(p, s, z, M, K, X[rows])
    got, w, ws = _gemm(ops, cuda, p, s, z, M, K, X)
    off = torch.zeros(R * M + 8, dtype=torch.float16, device=cuda)
    ops.gemm_w4a16(w, ws, _to_dev(X, cuda), off[2:2 + R * M].view(R, M))
    ws.check()
    one = off[2:2 + R * M].view(R, M).cpu().numpy()
    pairs, ref = (got[rows] != want).sum(), (one[rows] != want).sum()
    assert ref > 100 and pairs <= 1.3 * ref


@pytest.mark.parametrize("M,K,R", [(512, 512, 40), (512, 2048, 40),   # one CTA a tile, without and with its K split
                                   (1024, 1024, 300),                 # pairs, whole tiles
                                   (1024, 2048, 300), (384, 4096, 131),   # pairs, every tile split; an odd number of 128-output blocks
                                   (19200, 4096, 130)])               # pairs, a whole wave and a split tile
def test_gemm_epilogues(ops, orc, cuda, M, K, R):
    """The residual add and the GeLU act on the product as fp16: they equal the same operation on what the plain call stores (which
    the tests above hold to the oracle), the add bit by bit, the GeLU up to the last place of erf."""
    p, s, z = orc.gen_linear(44, M, K)
    X = orc.gen_normal_f16(44, orc.ACT, R * K).reshape(R, K)
    got, w, ws = _gemm(ops, cuda, p, s, z, M, K, X)
    rows = [0, R // 2, R - 1]
    y32, y16 = orc.gemm_w4a16(p, s, z, M, K, X[rows])
    _check(got[rows], y32, y16, f"{M}x{K} rows {R}", differ=0.05)
    old = orc.gen_normal_f16(45, orc.ACT, R * M).reshape(R, M)
    y = _to_dev(old, cuda)
    ops.gemm_w4a16_epilogue(w, ws, _to_dev(X, cuda), y, ops.cabi.EPI_RESIDUAL)
    assert np.array_equal(y.cpu().numpy().view(np.uint16), orc.add(old.ravel(), got.ravel()).reshape(R, M).view(np.uint16))
    ops.gemm_w4a16_epilogue(w, ws, _to_dev(X, cuda), y, ops.cabi.EPI_GELU)
    want = orc.gelu(got.ravel()).reshape(R, M)
    d = _ulp_diff(y.cpu().numpy(), want)
    # where 1 + erf cancels, a unit in the last place of erf (2^-24) times half the value is what is left of the result
    near = np.abs(y.cpu().numpy().astype(np.float32) - want.astype(np.float32)) <= 2.0 ** -23 * np.abs(got.astype(np.float32))
    assert ((d <= 1) | near).all()
    ws.check()
    assert ops.cabi.lib().qw3_gemm_w4a16_epilogue(w.h, y.data_ptr(), R, y.data_ptr(), ws.h, ops.cabi.EPI_ARGMAX, None) == ops.cabi.QW3_ERR_ARG


@pytest.mark.parametrize("M,K,R,integral", [
    (128, 1024, 129, True),     # row tiles of 32, four accumulators; one row in the last tile; half of the pair without outputs
    (640, 1024, 900, False),    # 64, four
    (896, 4096, 257, True),     # 96, three, K in six parts
    (384, 4096, 641, False),    # 128, three
    (896, 4096, 300, True),     # 160, three, K in seven parts
    (384, 4096, 513, True), (1152, 2048, 385, False), (3712, 512, 901, True)])   # 192, 224 and 256, two
def test_gemm_pairs_widths(ops, orc, cuda, M, K, R, integral):
    """The cuts that the times choose: every width of a row tile and number of accumulators, with rows that do not fill the last tile."""
    test_gemm_pairs_edges(ops, orc, cuda, M, K, R, integral)
