"""One row times a matrix in the decode-stream layout (decode_linear.cu) against sums in 64 bits: single tiles, ragged ones, rows of one unit up to the longest that
fits, every form of coefficients, and rows with outliers, whose small elements lose digits."""
import ctypes as C

import numpy as np
import pytest

from tests.util import bf16_to_f32, f32_to_bf16
from uzu_b200 import binding as B

pytestmark = [pytest.mark.gpu]


def _stream(codes, scales, coef, gps):
    """units of 16 rows x 512 nibbles: codes of rows g and g + 8 in lane order, then scales and zero points or biases in pairs of groups"""
    n, k = codes.shape
    tiles, units = -(-n // 16), -(-k // 512)
    q = np.zeros((tiles * 16, units * 512), np.uint8)
    q[:n, :k] = codes
    packed = (q[:, 0::2] | q[:, 1::2] << 4).reshape(tiles, 2, 8, units, 4, 4, 16)          # tile, half, g, unit, chunk, t, byte
    words = packed.transpose(0, 3, 1, 4, 2, 5, 6).reshape(tiles, units, 4096)
    pairs = np.zeros((tiles, units, 2, 2, 8, 4, 2), np.uint16)                             # scale / coef, half, g, t, pair
    for i, a in enumerate((scales, coef)):
        full = np.zeros((tiles * 16, units * gps), np.uint16)
        full[:n, :a.shape[1]] = a
        pairs[:, :, i, :, :, :gps // 2] = full.reshape(tiles, 2, 8, units, gps // 2, 2).transpose(0, 3, 1, 2, 4, 5)
    return np.concatenate([words, np.ascontiguousarray(pairs).view(np.uint8).reshape(tiles, units, 512)], -1)


def _operands(rng, n, k, group, method):
    codes = rng.integers(0, 16, (n, k), dtype=np.uint8)
    scales = f32_to_bf16(rng.uniform(0.002, 0.02, (n, k // group)).astype(np.float32))
    zero = rng.integers(0, 16, (n, k // group), dtype=np.uint8) if method == "zero" else np.full((n, k // group), 8, np.uint8)
    biases = f32_to_bf16((-bf16_to_f32(scales) * rng.integers(0, 16, scales.shape)).astype(np.float32))
    coef = biases if method == "mlx" else f32_to_bf16(zero.astype(np.float32))
    s = np.repeat(bf16_to_f32(scales).astype(np.float64), group, 1)
    c = np.repeat(bf16_to_f32(coef).astype(np.float64), group, 1)
    w = s * codes + c if method == "mlx" else s * (codes - c)
    size = s * codes + np.abs(c) * (1 if method == "mlx" else s)          # what the terms of a sum come to
    packed_zero = np.zeros((n, -(-(k // group) // 2)), np.uint8)
    packed_zero |= zero[:, 0::2]
    packed_zero[:, :zero[:, 1::2].shape[1]] |= zero[:, 1::2] << 4
    return codes, scales, packed_zero, biases, coef, w, size


def _run(ctx, n, k, group, method, x, ops, gated=False):
    codes, scales, zero, biases, coef = ops
    bufs = [ctx.upload(np.ascontiguousarray(a)) for a in (_stream(codes, scales, coef, 512 // group), codes[:, 0::2] | codes[:, 1::2] << 4, scales, zero, biases, x)]
    out = ctx.upload(np.zeros(n, np.float32))
    a = B.FusedLinearArgs(prologue=0, epilogue=int(gated), act_type=B.ACT_SILU, decode_stream=bufs[0].ptr)
    a.matmul = B.MatmulArgs(a=bufs[5].ptr, b=bufs[1].ptr, b_scales=bufs[2].ptr, b_zero_points=bufs[3].ptr if method == "zero" else 0, b_biases=bufs[4].ptr if method == "mlx" else 0,
                            d=out.ptr, b_prologue={"zero": B.B_SCALE_ZERO_POINT, "symmetric": B.B_SCALE_SYMMETRIC, "mlx": B.B_SCALE_BIAS}[method], b_mode=B.QMODE_U4, b_group_size=group,
                            b_transpose=1, ab_scale=1.0, m=1, n=n, k=k, weights_dt=B.DT_BF16, input_dt=B.DT_BF16, output_dt=B.DT_BF16 if gated else B.DT_F32)
    with ctx.command_buffer("decode-linear") as cmd:
        cmd.encode("uzu_fused_linear_encode", C.byref(a))
    return bf16_to_f32(out.numpy(np.uint16, (n // 2,))) if gated else out.numpy(np.float32, (n,))


def _row(rng, k, outliers):
    x = rng.standard_normal(k).astype(np.float32)
    if outliers:
        x[rng.integers(0, k, k // 64)] *= 2.0 ** rng.integers(-30, 24, k // 64)
    return f32_to_bf16(x)


@pytest.mark.parametrize("method", ["zero", "symmetric", "mlx"])
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("n,k", [(16, 512), (40, 1024), (2384, 512), (4752, 3584), (304, 14336), (48, 16384)])
def test_row_against_64_bits(ctx, n, k, group, method):
    rng = np.random.default_rng(n + k + group)
    *ops, w, size = _operands(rng, n, k, group, method)
    for outliers in (False, True):
        x = _row(rng, k, outliers)
        x64 = bf16_to_f32(x).astype(np.float64)
        got = _run(ctx, n, k, group, method, x, ops)
        # at most 6 roundings in a lane's sum of four groups, 2 in a quad's, C in a row's, each 2^-24 of what its terms come to, and digits cut off at
        # 2^-26 of a group's largest element
        top = np.repeat(np.abs(x64).reshape(-1, group).max(1), group)
        bound = (8 + 4 + -(-k // 512)) * 2.0 ** -24 * (size @ np.abs(x64)) + 2.0 ** -25 * (size @ top)
        assert (np.abs(got - w @ x64) <= bound).all()


@pytest.mark.parametrize("half,k", [(16, 512), (1200, 4096), (2384, 1024)])
def test_gated_rows(ctx, half, k):
    rng = np.random.default_rng(half + k)
    *ops, w, size = _operands(rng, 2 * half, k, 64, "zero")
    x = _row(rng, k, False)
    got = _run(ctx, 2 * half, k, 64, "zero", x, ops, gated=True)
    x64 = bf16_to_f32(x).astype(np.float64)
    y, sums = w @ x64, (12 - (-k // 512)) * 2.0 ** -24 * (size @ np.abs(x64)) + 2.0 ** -25 * size.sum(1) * np.abs(x64).max()      # as above
    up, gate, e_up, e_gate = y[:half], y[half:], sums[:half], sums[half:]
    act = gate / (1 + np.exp(-gate))
    want = up * act
    # roundings to bf16 (8 significant bits), 2^-8 each: up, the gate through a function of slope below 1.1, the function, the result
    e_up, e_gate = e_up + 2.0 ** -8 * np.abs(up), e_gate + 2.0 ** -8 * np.abs(gate)
    bound = np.abs(act) * e_up + 1.1 * np.abs(up) * e_gate + 1.1 * e_up * e_gate
    assert (np.abs(got - want) <= 1.01 * bound + 2.0 ** -7 * np.abs(want) + 1e-30).all()


def test_infinities_and_nans_stay_where_they_are(ctx):
    rng = np.random.default_rng(3)
    *ops, w, _ = _operands(rng, 64, 1024, 64, "zero")
    for bad in (np.inf, -np.inf, np.nan):
        x = bf16_to_f32(_row(rng, 1024, False))
        x[700] = bad
        assert np.isnan(_run(ctx, 64, 1024, 64, "zero", f32_to_bf16(x), ops)).all()      # codes - zero points of either sign times an infinity
    assert (_run(ctx, 64, 1024, 64, "zero", np.zeros(1024, np.uint16), ops) == 0).all()
