"""How the decode kernels deal their work out to CTAs, restated in Python and checked exhaustively: every unit or token is taken exactly
once, the contributors that a cut tile counts are those whose ranges meet it, no CTA uses a slot for two tiles.

* csrc/gemv_w4a16_tc.cu, DgRange: units (channel tile, quantisation group) of the W4A16 decode GEMM
* csrc/gemm_bf16_few.cu, GfRange: units (channel tile, 64 of K) of bf16 linears of 5 to 32 tokens, and which form serves a shape
* csrc/attention_mma.cu, at_share: blocks of 16 cached tokens of decode attention
"""
import random

import pytest

SMS = 148


def cdiv(a, b):
    return -(-a // b)


def check_ranges(tiles, per_tile, ctas, begin, owner):
    """begin(c): first unit of CTA c; owner(u): the CTA that holds the first or last unit u of a tile."""
    assert begin(0) == 0 and begin(ctas) == tiles * per_tile
    slots = {}
    meets = [[] for _ in range(tiles)]
    for c in range(ctas):
        u, end = begin(c), begin(c + 1)
        assert u <= end
        while u < end:
            tile = u // per_tile
            stop = min(end, (tile + 1) * per_tile)
            meets[tile].append(c)
            if not (u == tile * per_tile and stop == (tile + 1) * per_tile):
                slot = (c, 1 if c == owner(tile * per_tile) else 0)  # 1: the tile that the range ends inside
                assert slots.setdefault(slot, tile) == tile
            u = stop
    for tile, got in enumerate(meets):
        if len(got) > 1:
            assert got == list(range(owner(tile * per_tile), owner(tile * per_tile + per_tile - 1) + 1))


# ---- the W4A16 decode GEMM

def dg_launch(tiles, G):
    units = tiles * G
    grid, parts = max(1, min(SMS, units // 2)), 0
    if tiles <= SMS:
        p = max(1, min(SMS // tiles, G // 2))
        if cdiv(G, p) <= cdiv(units, grid) + 12:
            parts, grid = p, tiles * p
    return grid, parts


@pytest.mark.parametrize("G", [1, 2, 3, 7, 12, 16, 32, 56, 112])
def test_w4a16_decode_gemm(G):
    modes = set()
    for tiles in list(range(1, 330)) + [1002, 2048]:
        ctas, parts = dg_launch(tiles, G)
        total = tiles * G
        base, rem = divmod(total, ctas)
        assert ctas <= SMS
        modes.add(parts > 0)

        def begin(c):
            return c // parts * G + c % parts * G // parts if parts else c * base + min(c, rem)

        def owner(u):
            if parts:
                return u // G * parts + (parts - 1 if u % G else 0)
            cut = rem * (base + 1)
            return u // (base + 1) if u < cut else rem + (u - cut) // base
        check_ranges(tiles, G, ctas, begin, owner)
    assert modes == {True, False}


# ---- bf16 linears of a few tokens

CLUSTERS = {8: 16, 4: 32, 2: 74}  # clusters of so many CTAs that run side by side, at most (fewer where a GPC's last SMs make none up)


def in_whole(tiles, ctas):
    rounds = cdiv(tiles, ctas)
    return tiles * 20 >= ctas * 13 if rounds == 1 else rounds * ctas * 5 <= tiles * 6


def few_form(N, K, M, dual=False, stack=False):
    """'cluster', 'whole', 'cut' or 'gemv', by the host's rules (linear_simt.cu, gemm_bf16_few.cu)."""
    weights, tiles, ks, k = (2 if dual else 1) * N * K, cdiv(N, 128), cdiv(K, 64), (2 if dual else 1) * K
    pays = weights >= (5 if not stack and K < 4096 else 4) << 20 if M > 16 else weights >= 16 << 20 if M > 8 else M > 4 and K >= 4096 and weights >= 28 << 20
    if not pays or M > 32:
        return "gemv"
    if 2 * tiles <= SMS:
        cluster = 8
        while cluster > 2 and (cluster > ks or tiles > CLUSTERS[cluster]):
            cluster //= 2
        return "gemv" if ks < 2 or (not dual and M <= 16 and 8 * tiles < 3 * SMS and cluster == 2) else "cluster"
    ctas = tiles if tiles < SMS and in_whole(tiles, SMS) else SMS
    if in_whole(tiles, ctas):
        return "whole"
    least = (1024 if M > 16 else 2048 if M > 8 else 4096) if tiles < SMS else 0 if M > 16 else 1024
    return "gemv" if k <= least else "cut"


@pytest.mark.parametrize("ks", [2, 9, 16, 17, 32, 65, 112])
def test_bf16_ranges(ks):
    for tiles in list(range(SMS // 2 + 1, 700)) + [2000]:
        ctas = tiles if tiles < SMS and in_whole(tiles, SMS) else SMS
        whole = in_whole(tiles, ctas)

        def begin(c):
            return c * tiles // ctas * ks if whole else c * tiles * ks // ctas

        def owner(u):
            return ((u + 1) * ctas - 1) // (tiles * ks)
        check_ranges(tiles, ks, ctas, begin, owner)
        if whole:
            assert all(begin(c) % ks == 0 for c in range(ctas + 1))


def test_the_tests_of_a_few_tokens_reach_every_form():
    shapes = {"cluster": [(1000, 4200, 17), (4104, 4096, 31), (74 * 128, 1024, 32), (1536, 4096, 17), (2560, 2048, 32), (2048, 2560, 31), (4096, 4200, 9), (7168, 4096, 16),
                          (1000, 17000, 15), (4096, 7168, 5), (4096, 7168, 8)],
              "whole": [(12800, 1400, 17), (250 * 128, 544, 31), (14336, 4096, 8), (14336, 4096, 5)],
              "cut": [(75 * 128, 1800, 17), (95 * 128 + 8, 1800, 32), (149 * 128, 1024, 31), (219 * 128 + 40, 640, 17), (40000, 512, 32), (9600, 4096, 9), (149 * 128, 1400, 15), (10240, 4160, 6)],
              "gemv": [(2048, 2048, 32), (149 * 128, 1024, 9), (5120, 4096, 16), (4096, 4200, 8)]}
    for form, of in shapes.items():
        for s in of:
            assert few_form(*s) == form, (s, few_form(*s))
    for ff, M, form in [(149 * 128 + 8, 17, "cut"), (149 * 128 + 8, 9, "cut"), (12800, 20, "whole"), (80 * 128, 31, "cut"), (66 * 128 - 8, 12, "cluster")]:
        assert few_form(ff, 1032, M, dual=True, stack=True) == form


# ---- decode attention

def at_shares(lens, slots, nsplit, least=256, whole=512):
    blocks = [cdiv(n, 16) for n in lens]
    most = max(blocks)
    per = max(cdiv(sum(blocks), slots), cdiv(most, nsplit), least // 16)
    if most <= whole // 16:
        per = most
    while per < most and sum(cdiv(b, per) for b in blocks) > slots:
        per += max(1, per // 8)
    out = []
    for row, (n, b) in enumerate(zip(lens, blocks)):
        even = cdiv(b, cdiv(b, per)) if b else 1
        out += [(row, s, cdiv(b, even), s * even * 16, min(n, (s + 1) * even * 16)) for s in range(cdiv(b, even))]
    return out


def test_decode_attention_shares():
    rng = random.Random(2)
    for _ in range(3000):
        rows, kvh = int(2 ** rng.uniform(0, 8.1)), rng.choice([1, 2, 4, 8, 16, 32])
        top = int(2 ** rng.uniform(0, 15))
        lens = [rng.randint(1, top) for _ in range(rows)]
        slots = max(1, 2 * SMS // kvh)
        nsplit = max(1, min(cdiv(6 * SMS, rows * kvh), cdiv(max(lens), 64), 64))
        shares = at_shares(lens, slots, nsplit)
        assert len(shares) <= max(rows, min(slots, rows * nsplit))  # CTAs of a KV head that the launch has
        for row, n in enumerate(lens):
            mine = [s for s in shares if s[0] == row]
            assert [s[1] for s in mine] == list(range(mine[0][2])) and mine[0][2] <= nsplit
            assert mine[0][3] == 0 and mine[-1][4] == n
            assert all(a[4] == b[3] and b[3] % 16 == 0 for a, b in zip(mine, mine[1:])) and all(s[3] < s[4] for s in mine)
        if nsplit == 1 or max(lens) <= 512:  # the launch's short way: a CTA's row is its index
            assert shares == [(r, 0, 1, 0, n) for r, n in enumerate(lens)]
