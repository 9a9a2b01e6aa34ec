"""Index arithmetic of the thread-per-row pass kernel, on the CPU.

batch_rows_kernel (rtscan_b200/csrc/batch_rows.cuh; a part of kg groups of a
pass of G) keeps a pass's tables
in 128-byte lines whose slots hold copies of the columns of a group, lets
lane i of a quarter-warp visit the slots and 16-byte parts in the order
k ^ i, writes the row masks to a swizzled buffer, transposes 32-row tiles of
it in registers and writes the result words back as one line per query.
This test restates that arithmetic with numpy for every number of columns
and every pass shape, with all, some and
none of a pass's table positions in lines, and checks that

  * every table and buffer access stays inside its region,
  * every query's line holds the transposed masks computed directly,
  * the quarter-warp table loads (line layout) and mask stores and the
    warp's tile loads and result stores meet every bank at most once.
"""
import numpy as np
import pytest

FULL = 2**32 - 1


def groups_of(C, S):
    """(start, size) of every column's group: powers of two, largest first."""
    out, start, left = [], 0, C
    while left:
        size = S
        while size > left:
            size //= 2
        out += [(start, size)] * size
        start += size
        left -= size
    return out


def layout(C, kg, m, lines):
    """Byte offsets as rows_layout gives them for at most `lines` lines:
    first copies, bytes between copies, copies, rows past the lines, all."""
    S, row = 32 // kg, 4 * kg
    grp = groups_of(C, S)
    base, rep, nrep, over = [0] * C, [0] * C, [1] * C, [0] * C
    at, c = 0, 0
    while c < C:
        size = grp[c][1]
        for k in range(size):
            base[c + k], rep[c + k], nrep[c + k] = at + k * row, size * row, S // size
        at += min(max(m[c:c + size]) + 1, lines) * 128
        c += size
    for c in range(C):
        over[c] = at
        at += max(0, m[c] + 1 - lines) * row
    return base, rep, nrep, over, at


def transpose_octets(x):
    """The kernel's transpose on x[lane, 32] (x[8o + r]: row 8o + 7 - r)."""
    rot = lambda v, k: ((v << k) | (v >> (32 - k))) & FULL if k else v

    def perm(a, b, sel):
        by = [(a >> (8 * i)) & 255 for i in range(4)] + [(b >> (8 * i)) & 255 for i in range(4)]
        return sum(by[(sel >> (4 * i)) & 7] << (8 * i) for i in range(4))

    y = []
    for o in range(4):
        a = [rot(x[:, 8 * o + r], r) for r in range(8)]
        for d, m in ((1, 0x55555555), (2, 0x33333333), (4, 0x0F0F0F0F)):
            a = [(a[i] & m) | (a[(i + d) & 7] & (FULL ^ m)) for i in range(8)]
        y.append([rot(a[i], i) for i in range(8)])
    out = np.zeros_like(x)
    for i in range(8):
        u0, u1 = perm(y[1][i], y[0][i], 0x5140), perm(y[1][i], y[0][i], 0x7362)
        v0, v1 = perm(y[3][i], y[2][i], 0x5140), perm(y[3][i], y[2][i], 0x7362)
        out[:, (32 - i) & 31], out[:, 8 - i] = perm(v0, u0, 0x5410), perm(v0, u0, 0x7632)
        out[:, 16 - i], out[:, 24 - i] = perm(v1, u1, 0x5410), perm(v1, u1, 0x7632)
    return out


def one_per_bank(addr, lanes, banks, width):
    return all(len(set(q)) == lanes for q in (addr // width % banks).reshape(-1, lanes))


@pytest.mark.parametrize("lines", [1 << 20, 17, 0])
@pytest.mark.parametrize("G,kg", [(16, 8), (16, 4), (8, 8), (4, 4)])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8])
def test_rows_kernel_addresses(C, G, kg, lines):
    rng = np.random.default_rng(100 * C + G)
    g0 = 8 if G == 16 else 0  # the part's first group
    Q = kg // 4
    LQ = {2: 1, 1: 0}[Q]
    S, LS, RPT = 8 // Q, 3 - LQ, 32 // kg
    rows = 256 * RPT
    tiles = rows // 32
    m = [int(x) for x in rng.integers(0, 40, C)]
    grp = groups_of(C, S)
    base, rep, nrep, over, total = layout(C, kg, m, lines)
    mul, mul_over = 128 // G, 4 * kg // G
    tab = [rng.integers(0, 2**32, size=(m[c] + 1, G), dtype=np.uint64) for c in range(C)]
    tab_off, at = [], 0  # word offsets in the plan blob
    for c in range(C):
        tab_off.append(at)
        at += (m[c] + 1) * G
    smem = np.full(total // 4, 2**40, dtype=np.uint64)  # unwritten words are never masks
    for c in range(C):
        for pos in range(m[c] + 1):
            at = [base[c] + pos * 128 + r * rep[c] for r in range(nrep[c])] if pos < lines \
                else [over[c] + (pos - lines) * 4 * kg]
            for w in (a // 4 for a in at):
                assert w + kg <= smem.size
                assert np.all(smem[w:w + kg] == 2**40), "two table rows share words"
                smem[w:w + kg] = tab[c][pos, g0:g0 + kg]

    # phase A, all 256 threads
    tid = np.arange(256)
    lane, warp = tid & 31, tid >> 5
    hx, sb = lane & (Q - 1), (lane & 7) >> LQ
    pos = [rng.integers(0, m[c] + 1, size=rows) for c in range(C)]
    buf = np.full(8192, 2**40, dtype=np.uint64)
    mpos = (((tid & (S - 1)) * Q + (hx ^ ((tid >> LS) & (Q - 1)))) ^ warp) << 4
    for j in range(RPT):
        row = tid + 256 * j
        off = np.stack([tab_off[c] + pos[c][row] * G for c in range(C)])
        for s in range(Q):
            acc = np.full((256, 4), FULL, dtype=np.uint64)
            for k in range(C):
                start, size = grp[k]
                c = start + ((k - start) ^ (sb & (size - 1)))
                lc = np.array(base)[c] + np.array(rep)[c] * (sb >> size.bit_length() - 1) \
                    - np.array(tab_off)[c] * mul + (hx << 4)
                lim = np.array(tab_off)[c] + lines * G
                lo = np.array(over)[c] - lim * mul_over + (hx << 4)
                o = off[c, tid]
                addr = np.where(o < lim, o * mul + lc, o * mul_over + lo) ^ (s << 4)
                assert addr.min() >= 0 and addr.max() + 16 <= total and not np.any(addr & 15)
                if lines > max(m):
                    assert one_per_bank(addr, 8, 8, 16), "table loads of a quarter-warp share banks"
                for w in range(4):
                    acc[:, w] &= smem[addr // 4 + w]
            st = (tid // S) * 128 + j * (256 // S * 128) + (mpos ^ (s << 4))
            assert st.min() >= 0 and st.max() + 16 <= 32768
            assert one_per_bank(st, 8, 8, 16), "mask stores share banks"
            for w in range(4):
                buf[st // 4 + w] = acc[:, w]
    assert np.all(buf < 2**40)

    # phase B: lane (tile, group) reads its 32 mask words and writes its 32 result words
    h, oct_, tl, gl = warp & (Q - 1), warp >> LQ, lane >> 2, lane & 3
    tile, group = oct_ * 8 + tl, 4 * h + gl
    assert len({(int(t), int(g)) for t, g in zip(tile, group)}) == 256
    part = lambda r: ((r & (S - 1)) * Q + ((r >> LS) & (Q - 1))) << 4
    x = np.zeros((256, 32), dtype=np.uint64)
    for r in range(32):
        ld = (tile * 32 // S) * 128 + gl * 4 + (r // S) * 128 + (part(r) ^ ((h ^ tl) << 4))
        assert ld.min() >= 0 and ld.max() + 4 <= 32768
        assert one_per_bank(ld, 32, 32, 4), "mask loads of a warp share banks"
        want = np.full(256, FULL, dtype=np.uint64)
        for c in range(C):
            want &= tab[c][pos[c][32 * tile + r], g0 + group]
        assert np.array_equal(buf[ld // 4], want)
        x[:, (r & 24) | (7 - (r & 7))] = buf[ld // 4]
    x = transpose_octets(x)
    buf = np.full(8192, 2**40, dtype=np.uint64)  # every mask is in registers
    chunk = (2 * oct_ + (tl >> 2)) & 7
    region = h if Q == 2 else oct_ >> 2
    for j in range(32):
        st = region * 16384 + gl * 256 + (tl & 3) * 4 + 128 * (j & 1) + ((chunk ^ (2 * gl) ^ (j & 1)) << 4) \
            + (j >> 1) * 1024
        assert st.min() >= 0 and st.max() + 4 <= 32768
        assert one_per_bank(st, 32, 32, 4), "result stores of a warp share banks"
        buf[st // 4] = x[:, j]

    # phase C: line i holds query i's words, its 16-byte chunk c at c ^ (i % 8)
    mask = np.stack([np.bitwise_and.reduce([tab[c][pos[c], g0 + g] for c in range(C)])
                     for g in range(kg)], 1)  # [row, group]
    slots = set()
    for i in range(32 * kg):
        slot = (i & ~127) + 32 * ((i >> 1) & 3) + 2 * ((i & 127) >> 3) + (i & 1)
        slots.add(slot)
        bits = ((mask[:, slot >> 5] >> np.uint64(slot & 31)) & np.uint64(1)).reshape(tiles, 32)
        want = (bits << np.arange(31, -1, -1, dtype=np.uint64)).sum(1)
        got = []
        for part_ in range(tiles // 32):
            at = ((i if Q == 2 else 128 * part_ + i) * 128) // 4
            for c in range(8):
                got += list(buf[at + 4 * (c ^ (i & 7)):at + 4 * (c ^ (i & 7)) + 4])
        assert np.array_equal(np.array(got), want), i
    assert slots == set(range(32 * kg))
