"""The line arithmetic of the ragged tensor-core kernels (csrc/wmm_tc_ragged.cuh), restated: which elements of the band a tile
reads or writes, at which addresses, checked without a GPU for coverage, alignment and bounds against dense matrices."""
import random

import numpy as np
import pytest

TILE = 128


def _tile_mm(tr, M, Mo, w, off, lo, hi, b, t):
    W, r0, row0 = 2 * w + 1, t * TILE, b * M
    if not tr:
        brow = r0 - w + off
        m_lo, m_hi = 0, min(M - r0, TILE)
        klo, khi = max(lo - brow, 0), min(hi - brow, m_hi + 2 * w)
        a0 = (row0 + r0) * W
        kbeg = klo - ((klo + a0) & 1)
    else:
        r0 -= (row0 + w - off) & 1
        brow = r0 - off - w
        m_lo, m_hi = max(lo - r0, 0), min(min(Mo, hi) - r0, TILE)
        klo, khi = max(-brow, m_lo), min(M - brow, m_hi + 2 * w)
        a0 = (row0 + brow) * W + 2 * w
        kbeg = klo
    nch = (khi - kbeg + 63) // 64 if m_hi > m_lo and khi > klo else 0
    return r0, brow, m_lo, m_hi, klo, khi, kbeg, nch, a0


def _band_of(dense, w, off):
    """(M, Mo) -> the band (M, 2w+1), NaN where the position does not exist."""
    M, Mo = dense.shape
    band = np.full((M, 2 * w + 1), np.nan)
    for i in range(M):
        for j in range(2 * w + 1):
            p = i + j - w + off
            if 0 <= p < Mo:
                band[i, j] = dense[i, p]
    return band


def _cases():
    rng = random.Random(11)
    out = [(2, 33, 33, 4, 0, 0, 33), (1, 1, 1, 1, 0, 0, 1), (3, 50, 50, 90, 0, 0, 50), (2, 300, 300, 37, 0, 0, 300), (2, 257, 257, 64, 0, 0, 257)]
    for _ in range(12):
        M, w = rng.randint(1, 300), rng.randint(1, 140)
        Mo, off = rng.randint(1, 320), rng.randint(-30, 40)
        lo = rng.randint(0, Mo)
        out.append((rng.randint(1, 3), M, Mo, w, off, lo, rng.randint(lo, Mo)))
    return out


@pytest.mark.parametrize("case", _cases())
@pytest.mark.parametrize("tr", [False, True])
def test_band_lines_of_the_products(case, tr):
    B, M, Mo, w, off, lo, hi = case
    W = 2 * w + 1
    g = np.random.default_rng(0)
    dense = g.standard_normal((B, M, Mo))
    flat = np.concatenate([_band_of(dense[b], w, off) for b in range(B)]).ravel()
    rows_out = Mo if tr else M
    extra = 1 if tr and (((w - off) & 1) or ((M & 1) and B > 1)) else 0
    i, p = np.arange(M)[:, None], np.arange(Mo)[None, :]
    in_band = (np.abs(p - i - off) <= w) & (p >= lo) & (p < hi)
    for b in range(B):
        got = np.zeros((rows_out, M if tr else Mo))
        seen = np.zeros(rows_out, int)
        for t in range((rows_out + extra + TILE - 1) // TILE):
            r0, brow, m_lo, m_hi, klo, khi, kbeg, nch, a0 = _tile_mm(tr, M, Mo, w, off, lo, hi, b, t)
            seen[max(r0, 0):max(0, min(r0 + TILE, rows_out))] += 1
            for c in range(nch):
                k0 = kbeg + c * 64
                full = m_lo <= 0 and m_hi >= TILE and k0 >= klo and k0 + 64 <= khi and k0 >= TILE - 1 and k0 + 64 <= W
                for line in range(128):
                    if not tr:
                        m, addr = line, a0 + line * 2 * w + k0
                        e0, e1 = max(klo, m) - k0, (min(khi, m + W) - k0 if m < m_hi else 0)
                    else:
                        m0, k = line // 64 * 64, k0 + line % 64
                        addr = a0 + k * 2 * w + m0
                        e0, e1 = max(m_lo, k - W + 1) - m0, (min(m_hi, k + 1) - m0 if klo <= k < khi else 0)
                    assert addr % 2 == 0                       # aligned words
                    if full:
                        assert e0 <= 0 and e1 >= 64            # the unchecked path reads nothing it must not
                    e0, e1 = max(e0, 0), min(e1, 64)
                    if e0 >= e1:
                        continue
                    assert 0 <= addr + e0 and addr + e1 <= flat.size
                    vals = flat[addr + e0:addr + e1]
                    if not tr:
                        got[r0 + line, brow + k0 + e0:brow + k0 + e1] += vals
                    else:
                        got[r0 + m0 + e0:r0 + m0 + e1, brow + k] += vals
        assert (seen == 1).all()
        want = np.where(in_band, dense[b], 0.0)
        assert np.array_equal(got, want.T if tr else want)


@pytest.mark.parametrize("case", _cases())
def test_band_lines_of_band_nt(case):
    B, M, Mo, w, off, lo, hi = case
    W = 2 * w + 1
    written = np.zeros(B * M * W, int)
    for b in range(B):
        for t in range((M + TILE - 1) // TILE):
            r0, delta = t * TILE, (b * M) & 1
            for c in range((min(M - r0, TILE) + 2 * w + delta + 63) // 64):
                n0 = c * 64
                for quarter in range(4):
                    m0, rows = quarter * 32, min(32, M - r0 - quarter * 32)
                    if rows <= 0 or n0 + 63 < m0 + delta or n0 > m0 + 31 + delta + 2 * w:
                        continue
                    whole = rows == 32 and n0 >= m0 + 31 + delta and n0 + 64 <= m0 + delta + W
                    for u in range(rows):
                        m = m0 + u
                        line = (b * M + r0) * W - delta + m * 2 * w + n0
                        assert line % 2 == 0
                        e = np.arange(64)
                        j = n0 + e - m - delta
                        ok = (j >= 0) & (j < W)
                        assert ok.all() or not whole
                        assert np.array_equal(line + e[ok], (b * M + r0 + m) * W + j[ok])
                        assert np.array_equal(r0 - w + off - delta + n0 + e[ok], r0 + m + j[ok] - w + off)   # position of a column
                        written[line + e[ok]] += 1
    assert (written == 1).all()
