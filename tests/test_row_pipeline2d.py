"""Host replica of the 2-D kernels' row pipeline (Pipe2D, warp_item2d in
csrc/kernel2d.cuh): the column windows of every degree, the ring of row
buffers with its groups in flight and its kept rows, and the rows each copy
of the row code may be given. CPU only."""
import pytest


def pipe(R, B, assoc, terms, double, fma=True, div=False):
    W = 2 * R + 1
    row_instr = B * (terms * (2 if double else 4) * (1 if fma else 2) + (36 if div and not fma else 0) + 12) + 14
    rot = double or W * row_instr <= 1300
    slide = 800 // row_instr
    nph = W if rot else min(max(slide, 1), W - 1)
    pg = -(-(4 if double else 8) // nph)
    kg = -(-(B * R if assoc else 0) // nph)
    return W, nph, pg, kg, (pg + 1 + kg) * nph


@pytest.mark.parametrize("V", [4, 2])
@pytest.mark.parametrize("R", [1, 2, 3, 4])
@pytest.mark.parametrize("B", range(1, 9))
def test_windows_store_each_column_once_and_exactly(V, R, B):
    shift = (V - R % V) % V
    ml = -(-B * R // V) * V
    wout = (32 * V - ml - B * R) // V * V
    if wout <= 0:
        return
    for n in list(range(1, 70)) + [wout - 1, wout, wout + 1, 2 * wout, 2 * wout + 1, 1000, 4096]:
        d1 = n + 2 * R
        pitch = -(-(shift + d1 + 32 * V) // (8 * V)) * (8 * V)
        stored = [0] * d1
        for s in range(-(-n // wout)):
            cs, ws = R + s * wout, R + s * wout + shift - ml
            ce = min(cs + wout, d1 - R)
            assert ws % V == 0  # 16-byte aligned copies
            edge = ws - shift < R or ws - shift + 32 * V > d1 - R
            for lane in range(32):
                el = ws + lane * V
                col0 = el - shift
                whole = col0 >= cs and col0 + V <= ce
                for e in range(V):
                    c = col0 + e
                    copied = el >= 0 and el + V <= pitch
                    if 0 <= c < d1:
                        assert copied or not (cs - B * R <= c < ce + B * R)
                    if cs <= c < ce and (whole or edge):
                        stored[c] += 1
                        # b*r columns inside the window, or past the grid
                        assert c - B * R >= ws - shift or ws - shift <= 0
                        assert c + B * R < ws - shift + 32 * V
        assert stored == [0] * R + [1] * n + [0] * R, n


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("assoc", [False, True])
@pytest.mark.parametrize("R,terms", [(1, 5), (1, 9), (2, 9), (2, 25), (3, 13), (3, 49), (4, 17), (4, 81)])
@pytest.mark.parametrize("B", [1, 2, 3, 4, 6, 8])
def test_ring_holds_the_rows_that_are_read(R, terms, B, assoc, double):
    W, nph, pg, kg, nrows = pipe(R, B, assoc, terms, double)
    groups = nrows // nph
    for d0, sl in [(2 * R + 1, 1), (40, 3), (40, 40), (97, 16), (200, 31)]:
        for blk in range(-(-(d0 - 2 * R) // sl)):
            i0 = R + blk * sl
            i1 = min(i0 + sl, d0 - R)
            pstart, pend = max(0, i0 - B * R), min(d0, i1 + B * R)
            ng = -(-(i1 + B * R - pstart) // nph)
            ring = {}

            def request(g):
                for ph in range(nph):
                    row = pstart + g * nph + ph
                    if row < pend:
                        ring[g % groups * nph + ph] = row

            for g in range(pg):
                request(g)
            stored = []
            fast_lo = pstart if i0 >= B * R else (B + 1) * R
            fast_hi = 1 << 30 if i1 + B * R <= d0 else d0
            for g in range(ng):
                request(g + pg)
                pb, cur = pstart + g * nph, g % groups * nph
                interior = pb >= fast_lo and pb + nph <= fast_hi
                for ph in range(nph):
                    pp = pb + ph
                    if pp < pend:
                        assert ring[cur + ph] == pp
                    for lev in range(1, B + 1):
                        q, more = pp - lev * R, (B - lev) * R
                        if not i0 - more <= q <= i1 - 1 + more:
                            continue  # no output needs it
                        if interior:
                            assert R <= q < d0 - R
                        if assoc and 0 <= q < pend:  # its halo cells, from the ring
                            slot = cur + (q - pb)
                            assert ring[slot if slot >= 0 else slot + nrows] == q
                    if i0 <= pp - B * R < i1:
                        stored.append(pp - B * R)
            assert stored == list(range(i0, i1))
