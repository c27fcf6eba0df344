"""The partition of the line solves of one instance (linear_system_solvers_gb300/csrc/adi_split.hpp), compiled on
the host and checked without a GPU: chunks cover every row once, CTAs, tables and loads stay in
bounds, and host replays of the compositions (compose and k_wide_tdep in adi_wide.cuh) reproduce
the serial recurrences."""
import os
import subprocess
import tempfile

import numpy as np
import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "adi_split_t.cpp")
SMS = 152
MAX_CTA = 512
SHARED = 48 * 1024  # dynamic shared memory without an opt-in

SIZES = [(4, 4), (5, 9), (7, 18), (100, 50), (400, 200), (642, 256), (643, 257), (1026, 512), (1027, 513), (2050, 1024), (2051, 1025),
         (2600, 8), (6000, 200), (6000, 305), (6000, 307), (4096, 1000), (4096, 1218), (4096, 1219), (4096, 2048), (8, 20000), (300, 20000)]


class Split:
    def __init__(self, line):
        (self.L, self.PC, self.R, self.gs, self.tiles, self.groups, self.words, self.table) = (int(q) for q in line.split())


@pytest.fixture(scope="module")
def splits():
    out = os.path.join(tempfile.mkdtemp(), "adi_split_t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "linear_system_solvers_gb300", "csrc"), SRC, "-o", out],
                   check=True, capture_output=True, text=True)

    def ask(queries):
        res = subprocess.run([out], input="\n".join(" ".join(str(int(x)) for x in q) for q in queries), check=True,
                             capture_output=True, text=True)
        return [Split(ln) for ln in res.stdout.splitlines()]

    return ask


def pitch(ny):
    return (ny + 3) // 4 * 4


def counts(rows):
    """0 and the counts that lss_adi_line_chunks accepts for a line of `rows` rows."""
    return [0, 1] + [p for p in (2, 3, 7, 16, 31, 64, 100, 128) if rows >= 4 * p]


def both(splits, nx, ny, word=8, ps=0, pv=0):
    return splits([(0, nx - 2, ny - 2, ps, SMS, word, pitch(ny)), (1, ny, nx - 2, pv, SMS, word, nx)])


def cases(nx, ny):
    for word in (4, 8):
        for ps in counts(nx - 2):
            yield word, ps, 0
        for pv in counts(ny - 2):
            yield word, 0, pv


@pytest.mark.parametrize("nx,ny", SIZES)
def test_chunks_cover_every_row_once_and_ctas_fit(splits, nx, ny):
    for word, ps, pv in cases(nx, ny):
        s, v = both(splits, nx, ny, word, ps, pv)
        for sp, vec, rows, asked in ((s, False, nx - 2, ps), (v, True, ny, pv)):
            assert sp.R in ((4, 8, 16) if vec else (5, 8, 16))
            assert asked in (0, sp.PC)
            assert 1 <= sp.PC <= 128 and sp.L * sp.PC <= MAX_CTA
            assert (sp.tiles - 1) * sp.PC * sp.R < rows <= sp.tiles * sp.PC * sp.R
            first = [(tile * sp.PC + c) * sp.R for tile in range(sp.tiles) for c in range(sp.PC)]
            assert first == list(range(0, sp.tiles * sp.PC * sp.R, sp.R))  # consecutive chunks of R rows
            # composition: every chunk in one group, a thread of the line's own for every group
            assert sp.groups <= sp.PC and (sp.groups - 1) * sp.gs < sp.PC <= sp.groups * sp.gs
            assert sp.words == 2 * sp.L * (sp.PC + sp.groups)
            assert 2 * word * sp.words <= SHARED
            # k_wide_tdep: four entries of a map per chunk; of a group, or one per chunk
            assert 8 * sp.L * (4 * sp.PC + max(4 * sp.groups, sp.PC)) <= SHARED
        # the extrapolated row nx-1 is formed by the CTA that solved rows nx-2 and nx-3
        assert v.L >= 2


@pytest.mark.parametrize("nx,ny", SIZES)
def test_loads_stay_inside_their_line(splits, nx, ny):
    ld = pitch(ny)
    for word, ps, pv in cases(nx, ny):
        s, v = both(splits, nx, ny, word, ps, pv)
        # v stages: four columns from min(t, ld - 4), t a multiple of four; stores where t < ld
        t = np.arange(0, v.tiles * v.PC * v.R, 4)
        assert v.R % 4 == 0 and ld % 4 == 0
        col = np.minimum(t, ld - 4)
        assert np.all(col % 4 == 0) and col.min() >= 0 and col.max() + 3 < ld
        assert set(range(ny)) <= {int(c) + k for c in t[t < ld] for k in range(4)}
        # S stages: rows from min(t, nx-1), columns j-1, j, j+1 of an inner line (lanes outside are clamped)
        blocks = -(-(ny - 1) // s.L)
        lanes = np.arange(blocks * s.L)
        assert lanes.max() >= ny - 2  # every inner line has a lane
        j = np.clip(lanes, 1, ny - 2)
        assert j.min() - 1 >= 0 and j.max() + 1 <= ny - 1
        # v lines: rows nx-2 downwards, lanes below row 1 are clamped
        rows = nx - 2 - np.arange(-(-(nx - 2) // v.L) * v.L)
        assert set(range(1, nx - 1)) <= set(rows.tolist())


@pytest.mark.parametrize("nx,ny", [(4, 4), (100, 50), (400, 200), (4096, 2048), (400000, 8), (8, 400000), (1 << 28, 4), (4, 1 << 28)])
def test_product_tables_stay_below_the_line_tables(splits, nx, ny):
    """The products of a sweep take less than one line table of the same direction: a chunk has at least four
    rows and two values, and at most one row of chunks is padding."""
    s, v = both(splits, nx, ny)
    for sp, rows, stride in ((s, nx - 2, pitch(ny)), (v, ny, nx)):
        assert sp.table == sp.tiles * (2 * sp.PC + sp.groups) * stride
        padded = sp.tiles * sp.PC * sp.R
        assert rows <= padded < rows + sp.PC * sp.R
        assert sp.table <= padded * stride * 3 // sp.R


@pytest.mark.parametrize("rows,lines", [(7000, 6), (7000, 302), (7000, 306), (7000, 1216), (7000, 1217), (2049, 4000)])
def test_few_long_lines_take_more_chunks(splits, rows, lines):
    for word in (4, 8):
        (s,) = splits([(0, rows, lines, 0, SMS, word, lines)])
        if -(-lines // 8) > SMS:
            assert (s.L, s.PC) == (8, 32)
        else:
            assert s.PC == 128 and s.L == (2 if word == 8 and lines <= 2 * SMS else 4)


def compose(sp, end, a, value, fwd):
    """Incoming values of the chunks of one tile and the value entering the next, as `compose` forms them."""
    order = list(range(sp.PC)) if fwd else list(range(sp.PC - 1, -1, -1))  # chunk at each position of the sweep
    inside, pre, gb, ga = {}, {}, [], []
    for g in range(sp.groups):
        s, p = 0.0, 1.0
        for q in range(g * sp.gs, min((g + 1) * sp.gs, sp.PC)):
            c = order[q]
            inside[c], pre[c] = s, p
            s, p = a[c] * s + end[c], p * a[c]
        gb.append(s)
        ga.append(p)
    y, enter = value, []
    for g in range(sp.groups):
        enter.append(y)
        y = ga[g] * y + gb[g]
    return {c: pre[c] * enter[q // sp.gs] + inside[c] for q, c in enumerate(order)}, y


@pytest.mark.parametrize("rows,lines,vec,chunks", [(2, 2, 0, 0), (98, 48, 0, 0), (640, 9, 0, 0), (641, 9, 0, 0), (2600, 9, 0, 0), (7000, 2000, 0, 0),
                                                   (50, 98, 1, 0), (257, 9, 1, 0), (1300, 9, 1, 0), (300, 9, 0, 1), (300, 9, 0, 17), (300, 9, 1, 31)])
def test_composition_is_the_recurrence(splits, rows, lines, vec, chunks):
    (sp,) = splits([(vec, rows, lines, chunks, SMS, 8, lines)])
    r = np.random.default_rng(rows)
    n = sp.tiles * sp.PC * sp.R
    f, la = np.zeros(n), np.zeros(n)
    f[:rows], la[:rows] = r.standard_normal(rows), r.uniform(-0.99, 0.99, rows)
    for fwd in (True, False):
        want, y = np.zeros(n), 0.7
        for t in range(n) if fwd else range(n - 1, -1, -1):
            y = want[t] = f[t] - la[t] * y
        got, value = np.zeros(n), 0.7
        for tile in range(sp.tiles) if fwd else range(sp.tiles - 1, -1, -1):
            end, a = [], []
            rng = [[(tile * sp.PC + c) * sp.R + k for k in (range(sp.R) if fwd else range(sp.R - 1, -1, -1))] for c in range(sp.PC)]
            for c in range(sp.PC):
                y, p = 0.0, 1.0
                for t in rng[c]:
                    y, p = f[t] - la[t] * y, -la[t] * p
                end.append(y)
                a.append(p)
            enter, value = compose(sp, end, a, value, fwd)
            for c in range(sp.PC):
                y = enter[c]
                for t in rng[c]:
                    y = got[t] = f[t] - la[t] * y
        assert np.max(np.abs(got - want)) <= 1e-13 * max(1.0, np.max(np.abs(want)))


def pow2_inverse(*m):
    top = max(abs(x) for x in m)
    return 1.0 if top == 0.0 else 2.0 ** -(np.frexp(top)[1] - 1)


def tdep_factors(sp, M, P, Z, th, e):
    """la, gamma, 1/beta of rows 1..e as k_wide_tdep forms them: chunk maps of the Moebius recurrence
    beta_t = b_t - a_t c_{t-1} / beta_{t-1}, composed over groups, then every chunk's own rows."""
    la, gam, ib = np.zeros(e + 2), np.zeros(e + 2), np.zeros(e + 2)
    value = 1.0
    for tile in range(sp.tiles):
        maps, cins = [], []
        for c in range(sp.PC):
            t0 = 1 + (tile * sp.PC + c) * sp.R
            cin = cp = -th * P[t0 - 1] if 1 < t0 <= e + 1 else 0.0
            m = np.eye(2)
            for r in range(sp.R):
                t = t0 + r
                if t > e:
                    break
                b, ac = 1.0 + th * Z[t], -th * M[t] * cp
                cp = -th * P[t]
                m = np.array([[b, -ac], [1.0, 0.0]]) @ m
                if (r & 7) == 7 or r == sp.R - 1 or t == e:
                    m = m * pow2_inverse(*m.ravel())
            maps.append(m)
            cins.append(cin)
        before, groups = [], []
        for g in range(sp.groups):
            m = np.eye(2)
            for q in range(g * sp.gs, min((g + 1) * sp.gs, sp.PC)):
                before.append(m)
                m = maps[q] @ m
                m = m * pow2_inverse(*m.ravel())
            groups.append(m)
        x, y, enter = value, 1.0, []
        for m in groups:
            enter.append((x, y))
            x, y = m @ (x, y)
            sc = pow2_inverse(x, y, 0.0, 0.0)
            x, y = x * sc, y * sc
        value = x / y
        for c in range(sp.PC):
            bx, by = before[c] @ enter[c // sp.gs]
            g = cins[c] * by / bx if cins[c] != 0.0 else 0.0
            t0 = 1 + (tile * sp.PC + c) * sp.R
            for t in range(t0, min(t0 + sp.R, e + 1)):
                ib[t] = 1.0 / (th * M[t] * g + (1.0 + th * Z[t]))
                la[t] = -th * M[t] * ib[t]
                g = gam[t] = -th * P[t] * ib[t]
    return la, gam, ib


@pytest.mark.parametrize("e,lines", [(2, 5), (37, 5), (98, 48), (510, 254), (640, 20), (641, 20), (1025, 20), (2100, 20), (4500, 1300)])
@pytest.mark.parametrize("size", [0.01, 1.0])
def test_time_dependent_refactorisation_is_the_recurrence(splits, e, lines, size):
    (sp,) = splits([(0, e, lines, 0, SMS, 8, lines)])
    r = np.random.default_rng(e)
    th = 0.5
    M, P = size * r.uniform(0.0, 50.0, e + 2), size * r.uniform(0.0, 50.0, e + 2)
    Z = M + P + r.uniform(0.0, 1.0, e + 2)
    want = np.zeros((3, e + 2))
    g = 0.0
    for t in range(1, e + 1):
        beta = 1.0 + th * Z[t] + th * M[t] * g
        g = -th * P[t] / beta
        want[:, t] = -th * M[t] / beta, g, 1.0 / beta
    for got, w in zip(tdep_factors(sp, M, P, Z, th, e), want):
        assert np.max(np.abs(got[1:e + 1] - w[1:e + 1])) <= 1e-13 * np.max(np.abs(w))
