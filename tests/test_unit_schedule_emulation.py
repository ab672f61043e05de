"""CPU emulation of the unit schedules of csrc/lddmm_common.cuh and csrc/pairs_sym.cuh for every nesting of row blocks
and source tiles: symmetric self-sums with row blocks shorter or longer than a tile (SymGeom), two sources to a record
(SymStage), up to one and a half waves of CTAs; and the triangle of the energies (Units with kTriangle), whose sources are
the targets first. Every ordered pair is credited exactly once, every index stays in its buffer."""
import numpy as np
import pytest

from test_scratch_sizes import _cta_of, _max_slots, _row_off, _tri


def _start(c, W, C):
    return c * W // C


def _row_of(u, nblk, TT, TPB, B):
    return max(i for i in range(nblk) if _row_off(i, TT, TPB, B) <= u)


class Geo:
    def __init__(self, TPB, B):
        self.TPB, self.B, self.K = TPB, B, max(TPB, B)
        self.span, self.share = max(1, B // TPB), max(1, TPB // B)

    def first_tile(self, i):
        return i * self.span if self.B >= self.TPB else i // self.share

    def col_first(self, J):
        return self.share * _tri(J)


@pytest.mark.parametrize('TPB', [64, 128])
@pytest.mark.parametrize('B', [32, 64, 128, 256, 768])
@pytest.mark.parametrize('wave', [5, 60, 444])
def test_symmetric_units(TPB, B, wave):
    G = Geo(TPB, B)
    for n in (1, 31, 33, 129, 700, 1409):
        nblk, TT = -(-n // B), -(-n // TPB)
        U = _row_off(nblk, TT, TPB, B)
        C = U if 2 * U < 3 * wave else wave
        S = _max_slots(TT, U, C)
        Kf = np.random.default_rng(n).normal(size=(n, n))
        Kf = Kf + Kf.T
        v = np.random.default_rng(B).normal(size=n)
        row_ws = np.full((S, n), np.nan)
        col_ws = np.full(G.col_first(-(-n // G.K)) * G.K, np.nan)
        credited = np.zeros((n, n), dtype=np.int64)
        for cta in range(C):
            u, u_end = _start(cta, U, C), _start(cta + 1, U, C)
            i = _row_of(u, nblk, TT, TPB, B) if u < u_end else 0
            while u < u_end:
                off = _row_off(i, TT, TPB, B)
                first = G.first_tile(i)
                cnt = TT - first
                t0, t1 = u - off, min(cnt, u_end - off)
                slot = cta - _cta_of(off, U, C)
                assert 0 <= slot < S
                rows = np.arange(i * B, min(i * B + B, n))
                acc = np.zeros(len(rows))
                for tt in range(t0, t1):
                    t = first + tt
                    src = np.arange(t * TPB, min(t * TPB + TPB, n))
                    acc += Kf[np.ix_(rows, src)] @ v[src]
                    credited[np.ix_(rows, src)] += 1
                    if tt >= G.span:                                   # past the row block's own superblock
                        J = t * TPB // G.K
                        base = (G.col_first(J) + i) * G.K + t * TPB - G.K * J
                        assert i < J * G.share and np.isnan(col_ws[base + src - t * TPB]).all()
                        col_ws[base + src - t * TPB] = Kf[np.ix_(rows, src)].T @ v[rows]
                        credited[np.ix_(src, rows)] += 1
                row_ws[slot, rows] = acc
                u += t1 - t0
                i += 1
        assert (credited == 1).all()
        out = np.zeros(n)
        for k in range(n):                                             # the epilogue
            b, J = k // B, k // G.K
            nslot = _cta_of(_row_off(b + 1, TT, TPB, B) - 1, U, C) - _cta_of(_row_off(b, TT, TPB, B), U, C) + 1
            cols = [(G.col_first(J) + q) * G.K + k - J * G.K for q in range(J * G.share)]
            out[k] = row_ws[:nslot, k].sum() + col_ws[cols].sum()
        assert np.allclose(out, Kf @ v, rtol=0, atol=1e-11 * n)


@pytest.mark.parametrize('TPB,B', [(128, 1024), (128, 512), (128, 256), (128, 128), (128, 64), (128, 32)])
@pytest.mark.parametrize('wave', [5, 444])
def test_energy_triangle_units(TPB, B, wave):
    """sum over k, l < self of f(k, l) (symmetric) and over the other sources, from the units of the triangle with weight
    1 on a row block's own superblock and 2 beyond it."""
    G = Geo(TPB, B)
    for n, other in ((1, 0), (1, 1), (130, 0), (130, 7), (700, 300), (1100, 1409)):
        ts = -(-n // TPB)
        TT = ts + -(-other // TPB)
        gx = -(-n // B)
        W = _row_off(gx, TT, TPB, B)
        C = min(W, wave)
        S = _max_slots(TT, W, C)
        f = np.random.default_rng(n).normal(size=(n, n + other))
        f[:, :n] += f[:, :n].T.copy()
        total, units = 0.0, 0
        weight = np.zeros((n, n + other))
        for cta in range(C):
            u, u_end = _start(cta, W, C), _start(cta + 1, W, C)
            tb = _row_of(u, gx, TT, TPB, B) if u < u_end else 0
            while u < u_end:
                off, first = _row_off(tb, TT, TPB, B), G.first_tile(tb)
                j0, j1 = first + u - off, first + min(TT - first, u_end - off)
                assert 0 <= cta - _cta_of(off, W, C) < S
                rows = np.arange(tb * B, min(tb * B + B, n))
                for j in range(j0, j1):
                    units += 1
                    w = 1.0
                    if j < ts:
                        src = np.arange(j * TPB, min(j * TPB + TPB, n))
                        if j >= first + G.span:
                            w = 2.0
                    else:
                        src = n + np.arange((j - ts) * TPB, min((j - ts) * TPB + TPB, other))
                    total += w * f[np.ix_(rows, src)].sum()
                    weight[np.ix_(rows, src)] += w
                u += j1 - j0
                tb += 1
        assert units == W
        pair = weight[:, :n] + weight[:, :n].T
        assert (pair == 2).all() and (weight[:, n:] == 1).all()
        assert np.isclose(total, f.sum(), rtol=0, atol=1e-9 * f.size)


@pytest.mark.parametrize('TPB,R', [(128, 32), (128, 16), (64, 32)])
def test_records_of_two_sources(TPB, R):
    """FP32 staging: source t of a tile is half (t / R) mod 2 of record (t / 2R) R + t mod R. The ring of R lanes brings
    record (lane + s) mod R of its chunk to a lane at step s; a column sum that moves to the lane before after every step
    has met every lane of its half warp when it is back."""
    where = {}
    for t in range(TPB):
        rec, half = t // (2 * R) * R + t % R, t // R & 1
        assert (rec, half) not in where
        where[rec, half] = t
    assert sorted(where) == [(r, h) for r in range(TPB // 2) for h in (0, 1)]
    for chunk in range(TPB // (2 * R)):
        lanes = np.arange(32)
        nxt = ((lanes + 1) & (R - 1)) | (lanes & ~(R - 1))            # ring_next: a lane takes its value from there
        col = [dict() for _ in lanes]                                   # per lane: record -> lanes met
        for s in range(R):
            rec = chunk * R + ((lanes + s) & (R - 1))
            for l in lanes:
                assert not col[l] or set(col[l]) == {rec[l]}
                col[l].setdefault(rec[l], []).append(l)
            col = [col[nxt[l]] for l in lanes]
        for l in lanes:
            rec = chunk * R + (l & (R - 1))
            assert list(col[l]) == [rec] and sorted(col[l][rec]) == [k for k in lanes if (k & ~(R - 1)) == (l & ~(R - 1))]
            # whole tiles: sums of chunk `chunk` at 64 chunk + lane and + 32; split: lane l < 16 gives source l, else l
            if R == 32:
                assert (where[rec, 0], where[rec, 1]) == (chunk * 64 + l, chunk * 64 + 32 + l)
            else:
                assert where[rec, int(l >= 16)] == chunk * 32 + l
