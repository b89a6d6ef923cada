"""One row times a matrix in the decode-stream layout (decode_linear.cu) against sums in 64 bits: single tiles, ragged ones, rows of one unit up to the longest that
fits, both code widths, every form of coefficients, the norm and the gate in front of the product, and rows with outliers, whose small elements lose digits."""
import ctypes as C

import numpy as np
import pytest

from tests.util import bf16_to_f32, f32_to_bf16
from uzu_b200 import binding as B

pytestmark = [pytest.mark.gpu]


def _stream(codes, scales, coef, bits, gps):
    """units of 16 rows x 512 nibbles: codes of rows g and g + 8 in lane order, then scales and zero points or biases in pairs of groups"""
    n, k = codes.shape
    unit_k = 512 * 4 // bits
    tiles, units = -(-n // 16), -(-k // unit_k)
    q = np.zeros((tiles * 16, units * unit_k), np.uint8)
    q[:n, :k] = codes
    packed = (q[:, 0::2] | q[:, 1::2] << 4 if bits == 4 else q).reshape(tiles, 2, 8, units, 4, 4, 16)          # tile, half, g, unit, chunk, t, byte
    words = packed.transpose(0, 3, 1, 4, 2, 5, 6).reshape(tiles, units, 4096)
    pairs = np.zeros((tiles, units, 2, 2, 8, 4, 2), np.uint16)                             # scale / coef, half, g, t, pair
    for i, a in enumerate((scales, coef)):
        full = np.zeros((tiles * 16, units * gps), np.uint16)
        full[:n, :a.shape[1]] = a
        pairs[:, :, i, :, :, :gps // 2] = full.reshape(tiles, 2, 8, units, gps // 2, 2).transpose(0, 3, 1, 2, 4, 5)
    return np.concatenate([words, np.ascontiguousarray(pairs).view(np.uint8).reshape(tiles, units, 512)], -1)


def _operands(rng, n, k, group, method, bits=4):
    most = 1 << bits
    codes = rng.integers(0, most, (n, k), dtype=np.uint8)
    scales = f32_to_bf16((rng.uniform(0.002, 0.02, (n, k // group)) * 16 / most).astype(np.float32))
    zero = rng.integers(0, most, (n, k // group), dtype=np.uint8) if method == "zero" else np.full((n, k // group), most // 2, np.uint8)
    biases = f32_to_bf16((-bf16_to_f32(scales) * rng.integers(0, most, scales.shape)).astype(np.float32))
    coef = biases if method == "mlx" else f32_to_bf16(zero.astype(np.float32))
    s = np.repeat(bf16_to_f32(scales).astype(np.float64), group, 1)
    c = np.repeat(bf16_to_f32(coef).astype(np.float64), group, 1)
    w = s * codes + c if method == "mlx" else s * (codes - c)
    size = s * codes + np.abs(c) * (1 if method == "mlx" else s)          # what the terms of a sum come to
    packed_zero = zero
    if bits == 4:
        packed_zero = np.zeros((n, -(-(k // group) // 2)), np.uint8)
        packed_zero |= zero[:, 0::2]
        packed_zero[:, :zero[:, 1::2].shape[1]] |= zero[:, 1::2] << 4
    return codes, scales, packed_zero, biases, coef, w, size


def _run(ctx, n, k, group, method, x, ops, gated=False, bits=4, fused=None):
    """fused: fields of the call beside the product; arrays among them are uploaded. With a "shortcut_out", that row comes back as well."""
    codes, scales, zero, biases, coef = ops
    packed = codes[:, 0::2] | codes[:, 1::2] << 4 if bits == 4 else codes
    bufs = [ctx.upload(np.ascontiguousarray(a)) for a in (_stream(codes, scales, coef, bits, 2048 // bits // group), packed, scales, zero, biases, x)]
    out = ctx.upload(np.zeros(n, np.float32))
    fields = {name: ctx.upload(v) if isinstance(v, np.ndarray) else v for name, v in (fused or {}).items()}
    a = B.FusedLinearArgs(**{"prologue": 0, "epilogue": int(gated), "act_type": B.ACT_SILU, "decode_stream": bufs[0].ptr,
                             **{name: v.ptr if hasattr(v, "ptr") else v for name, v in fields.items()}})
    a.matmul = B.MatmulArgs(a=0 if fused else bufs[5].ptr, b=bufs[1].ptr, b_scales=bufs[2].ptr, b_zero_points=bufs[3].ptr if method == "zero" else 0, b_biases=bufs[4].ptr if method == "mlx" else 0,
                            d=out.ptr, b_prologue={"zero": B.B_SCALE_ZERO_POINT, "symmetric": B.B_SCALE_SYMMETRIC, "mlx": B.B_SCALE_BIAS}[method], b_mode=B.QMODE_U4 if bits == 4 else B.QMODE_U8,
                            b_group_size=group, b_transpose=1, ab_scale=1.0, m=1, n=n, k=k, weights_dt=B.DT_BF16, input_dt=B.DT_BF16, output_dt=B.DT_BF16 if gated else B.DT_F32)
    with ctx.command_buffer("decode-linear") as cmd:
        if bits == 4:
            cmd.encode("uzu_fused_linear_encode", C.byref(a))
        else:                    # (that entry takes 4-bit weights only)
            assert ctx.lib.uzu_debug_fused_linear_encode(cmd.h, C.byref(a)) == 1
    got = bf16_to_f32(out.numpy(np.uint16, (n // 2,))) if gated else out.numpy(np.float32, (n,))
    return (got, fields["shortcut_out"].numpy(np.uint16, (k,))) if fused and "shortcut_out" in fused else got


def _row(rng, k, outliers):
    x = rng.standard_normal(k).astype(np.float32)
    if outliers:
        x[rng.integers(0, k, k // 64)] *= 2.0 ** rng.integers(-30, 24, k // 64)
    return f32_to_bf16(x)


def _bound(x64, size, k, group, bits):
    """at most 6 roundings in a lane's sum of four groups, 2 in a quad's, C in a row's, each 2^-24 of what its terms come to, and digits cut off at 2^-26 of a group's largest
    element; with bytes a pair of digits' sum has up to 28 bits and is rounded to 24 as well, 2^-24 of twice the largest element's terms"""
    top = np.repeat(np.abs(x64).reshape(-1, group).max(1), group)
    return (8 + 4 + -(-k * bits // 2048)) * 2.0 ** -24 * (size @ np.abs(x64)) + (2.0 ** -25 + (2.0 ** -23 if bits == 8 else 0)) * (size @ top)


FORMS = [(4, 64, "zero"), (4, 64, "symmetric"), (4, 64, "mlx"), (4, 128, "zero"), (4, 128, "symmetric"), (4, 128, "mlx"), (8, 64, "zero"), (8, 64, "symmetric"), (8, 64, "mlx")]


@pytest.mark.parametrize("bits,group,method", FORMS)
@pytest.mark.parametrize("n,k", [(16, 512), (40, 1024), (2384, 512), (4752, 3584), (304, 14336), (48, 16384)])
def test_row_against_64_bits(ctx, n, k, group, method, bits):
    rng = np.random.default_rng(n + k + group)
    k = k * 4 // bits
    *ops, w, size = _operands(rng, n, k, group, method, bits)
    for outliers in (False, True):
        x = _row(rng, k, outliers)
        x64 = bf16_to_f32(x).astype(np.float64)
        got = _run(ctx, n, k, group, method, x, ops, bits=bits)
        assert (np.abs(got - w @ x64) <= _bound(x64, size, k, group, bits)).all()


def _bf16(x):
    return bf16_to_f32(f32_to_bf16(np.asarray(x, np.float32)))


# rows of one piece a thread, of two, and longer ones, whose later pieces wait in the place of their own digits (4-bit rows above 8192, 8-bit ones above 4096)
@pytest.mark.parametrize("bits,group,method", FORMS)
@pytest.mark.parametrize("nibbles", [2048, 32768, 34816, 49152])
@pytest.mark.parametrize("prologue,add,full", [(1, True, False), (1, False, True), (3, False, False)])
def test_rows_with_a_prologue(ctx, bits, group, method, nibbles, prologue, add, full):
    n, k = 80, nibbles // bits
    rng = np.random.default_rng(nibbles + bits)
    *ops, w, size = _operands(rng, n, k, group, method, bits)
    x, other = _row(rng, k, False), _row(rng, k, False)
    a, b = bf16_to_f32(x), bf16_to_f32(other)
    if prologue == 1:
        scales = rng.uniform(0.5, 1.5, k).astype(np.float32)
        row = _bf16(a + b) if add else a
        got, kept = _run(ctx, n, k, group, method, x, ops, bits=bits,
                         fused=dict(prologue=1, norm_input=x, norm_shortcut_in=other, norm_scales=scales, shortcut_out=np.zeros(k, np.uint16), norm_epsilon=1e-5, norm_scale_offset=0.25,
                                    norm_residual_add=int(add), norm_full_layer=int(full)))
        assert np.array_equal(kept, f32_to_bf16(row))
        inv = np.float32(1 / np.sqrt(np.mean(row.astype(np.float64) ** 2) + 1e-5))
        want = _bf16(row * inv * (scales + np.float32(0.25))) if full else _bf16(_bf16(row * inv) * _bf16(scales + np.float32(0.25)))
    else:
        got = _run(ctx, n, k, group, method, x, ops, bits=bits, fused=dict(prologue=3, sg_attn=x, sg_gate=other))
        want = _bf16(a * (1 / (1 + np.exp(-b.astype(np.float64)))).astype(np.float32))
    x64 = want.astype(np.float64)
    # the root and the gate may differ in the last bits of f32 (2^-22): one element in 2^12 is then rounded to its neighbour, of a quarter and an eighth of a per cent; 12 of them
    # at most (expected: 3 of the longest rows)
    flips = 12 * 2.0 ** -7 * np.abs(x64).max() * np.abs(w).max(1)
    assert (np.abs(got - w @ x64) <= _bound(x64, size, k, group, bits) + flips).all()
    assert np.median(np.abs(got - w @ x64)) <= np.median(_bound(x64, size, k, group, bits)) + 2.0 ** -8 * np.abs(w).max() * np.abs(x64).max()


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


def test_a_row_that_is_not_finite(ctx):
    """An infinity or a NaN makes NaN of every output, as in the kernel before: codes and the zero point, which multiplies the row's sum, are taken apart."""
    rng = np.random.default_rng(3)
    *ops, w, _ = _operands(rng, 64, 1024, 64, "zero")
    for bad in (np.inf, -np.inf, np.nan):
        x = bf16_to_f32(_row(rng, 1024, False))
        x[700] = bad
        assert np.isnan(_run(ctx, 64, 1024, 64, "zero", f32_to_bf16(x), ops)).all()
    assert (_run(ctx, 64, 1024, 64, "zero", np.zeros(1024, np.uint16), ops) == 0).all()
