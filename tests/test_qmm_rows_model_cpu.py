"""Lane-level model of the few-row quantised product (uzu_b200/csrc/qmm_rows.cu), checked on the CPU by enumeration: which codes a lane reads, the order
its activations lie in, the fragments of mma.sync.m16n8k16 (A rows g / g + 8, B column g = activation row g, D columns 2t / 2t + 1), integer codes less
the zero point's nibbles, and a group's scale on its sum. It must give sum_k x[k] * scale[g(k)] * (code[k] - zp[g(k)]) for every (feature, row) of a step."""
import numpy as np
import pytest


def fragment_order(x, bits):
    """8 neighbouring activations as the four pairs of a 16-byte piece"""
    pairs = ((0, 4), (1, 5), (2, 6), (3, 7)) if bits == 4 else ((0, 2), (1, 3), (4, 6), (5, 7))
    return [(x[i], x[j]) for i, j in pairs]


def code_pairs(codes, zero, bits):
    """the four pairs a lane forms from 8 codes: nibbles i and i + 4 of a word, or bytes (0, 2) and (1, 3) of two words, as 16 (high - zh) + (low - zl)"""
    if bits == 4:
        d = [c - zero for c in codes]
        return [(d[i], d[i + 4]) for i in range(4)]
    d = [16 * ((c >> 4) - (zero >> 4)) + ((c & 15) - (zero & 15)) for c in codes]
    return [(d[0], d[2]), (d[1], d[3]), (d[4], d[6]), (d[5], d[7])]


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("group", [64, 128])
def test_a_step_is_the_dequantised_dot_product(bits, group):
    rng = np.random.default_rng(bits + group)
    K = 512 if bits == 4 else 256
    groups = K // group
    codes = rng.integers(0, 1 << bits, (16, K))
    scales, zeros = rng.uniform(0.01, 0.3, (16, groups)), rng.integers(0, 1 << bits, (16, groups))
    x = rng.uniform(-0.5, 0.5, (8, K))
    items = [[fragment_order(x[r, 8 * i:8 * i + 8], bits) for i in range(K // 8)] for r in range(8)]
    used = np.zeros((16, K), int)
    acc = np.zeros((16, 8))
    for gq in range(groups):
        d = np.zeros((16, 8))
        for part in range(group // 64):
            q = gq * (group // 64) + part
            for w in range(2):
                for feature in range(16):                    # A rows: lanes g = feature % 8 feed a (row g) and b (row g + 8)
                    for row in range(8):                     # B columns: lanes g = row
                        for t in range(4):                   # the quad's lanes hold the 16 k of two products
                            first = 64 * q + 16 * t + 8 * w  # 8 or 16 bytes of shared memory per lane: its 16 codes, word(s) w
                            a = code_pairs([int(c) for c in codes[feature, first:first + 8]], int(zeros[feature, gq]), bits)
                            b = items[row][8 * q + 2 * t + w]
                            d[feature, row] += sum(p[0] * v[0] + p[1] * v[1] for p, v in zip(a, b))
                            if row == 0:
                                used[feature, first:first + 8] += 1
        acc += scales[:, gq, None] * d
    assert (used == 1).all()
    want = np.einsum("fk,rk->fr", np.repeat(scales, group, 1) * (codes - np.repeat(zeros, group, 1)), x)
    np.testing.assert_allclose(acc, want, rtol=1e-12, atol=1e-12)


def test_shared_memory_reads_fall_on_all_banks():
    """Codes at pitches of 288 (8 bytes a lane, 16 lanes at a time) and 320 bytes (16 bytes, 8 lanes); activation rows an odd number of 16-byte pieces apart."""
    lanes = [(lane >> 2, lane & 3) for lane in range(32)]
    for lo in (0, 16):
        banks = {(g * 288 + t * 8 + b) // 4 % 32 for g, t in lanes[lo:lo + 16] for b in (0, 4)}
        assert len(banks) == 32
    for lo in range(0, 32, 8):
        assert len({(g * 320 + t * 16 + b) // 4 % 32 for g, t in lanes[lo:lo + 8] for b in (0, 4, 8, 12)}) == 32
        for pieces in (64, 256, 448, 32):
            assert len({(g * (pieces + 1) + 2 * t) % 8 for g, t in lanes[lo:lo + 8]}) == 8


@pytest.mark.parametrize("warps", [12])
def test_runs_of_a_column_meet(warps):
    """Every (tile, step) belongs to one warp; a tile that several warps share is begun by one, and the following ones add to it in order."""
    for tiles in (1, 2, 5, 11, 105):
        for steps in (1, 2, 7, 28):
            for whole in (False, True):
                at = [w * tiles // warps * steps if whole else w * tiles * steps // warps for w in range(warps + 1)]
                assert at[0] == 0 and at[-1] == tiles * steps and at == sorted(at)
                for tile in range(tiles):
                    begun = [w for w in range(warps) if at[w] <= tile * steps < at[w + 1]]
                    assert len(begun) == 1
                    sharers = [w for w in range(warps) if max(at[w], tile * steps) < min(at[w + 1], (tile + 1) * steps)]
                    assert sharers[0] == begun[0] and (not whole or len(sharers) == 1)
                    for w in sharers[1:]:                     # one slot per warp: it is in the middle of no other tile
                        assert at[w] // steps == tile
