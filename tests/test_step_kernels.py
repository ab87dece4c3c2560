"""The step's kernels at the sizes where their layouts change: particle counts on and
beside the blocks' edges, handles below and above the size where blocks of few particles
give way to full ones, and the integer forms of the integrator's FP64 operations."""
import math
import random
import struct

import numpy as np
import pytest

from oracle_bridge import Oracle
from systems import golden_inputs, load
from tis_gb300 import PREC_FP64, PREC_MIXED, STATE_NAMES, Engine


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


@pytest.mark.parametrize("box", [51.3, 65.0, 200.0, 277.5, 350.0, 600.0, 1000.0, 2048.0, 4096.0])
def test_position_floor_by_integers(box):
    """fix_position's arithmetic (constants as tis_create forms them) against floor of the
    rounded FP64 product, over the box, its image, small and negative coordinates and the
    neighbours of exact multiples."""
    rng = random.Random(int(box))
    qinv = 4294967296.0 / box
    e2l, eq = math.frexp(2.0 * box)[1], math.frexp(qinv)[1]
    q, hi2l, sh, fb = int(math.ldexp(qinv, 64 - eq)), _bits(2.0 * box) >> 32, 1022 + e2l, 64 - eq - e2l - 1
    assert 28 <= fb <= 30 and q < 2 ** 64
    fast = 0
    for k in range(20000):
        kind = k % 4
        x = rng.uniform(0, 2 * box) if kind == 0 else rng.uniform(0, box) * 2.0 ** -rng.randint(0, 60) if kind == 1 else \
            math.nextafter(rng.randrange(2 ** 32) / qinv, rng.choice([-1e9, 1e9])) if kind == 2 else rng.uniform(-box, 0)
        want = math.floor(x * qinv) % 2 ** 32
        b = _bits(x)
        hi = b >> 32
        if hi < hi2l:
            s = sh - (hi >> 20)
            assert s >= 0
            m = ((((hi & 0xFFFFF) | 0x100000) << 32) | (b & 0xFFFFFFFF)) << 10
            v = ((m >> s if s < 64 else 0) * q) >> 64
            if (v & ((1 << fb) - 1)) < (1 << fb) - (1 << (fb - 20)):
                fast += 1
                assert (v >> fb) % 2 ** 32 == want, (x, box)
    assert fast > 5000


def test_fixed_point_to_double_by_integers():
    """fix_to_double's arithmetic against the conversion, up to the 53 bits it covers."""
    rng = random.Random(7)
    for v in [0, 1, -1, 2 ** 53 - 1, 1 - 2 ** 53] + [rng.randrange(-2 ** n, 2 ** n + 1) for n in range(1, 53) for _ in range(200)]:
        m = abs(v)
        b = 0
        if m:
            z = 64 - m.bit_length()
            b = ((((m << z) << 1) & (2 ** 64 - 1)) >> 12) | ((1086 - z) << 52)
        assert b | ((1 << 63) if v < 0 else 0) == _bits(float(v)), v


@pytest.mark.gpu
@pytest.mark.parametrize("n_cl,n_k", [(0, 0), (27, 1), (27, 2), (261, 406), (261, 407), (261, 408)])
def test_particle_counts_at_block_edges(n_cl, n_k):
    """Stochastic FP64 steps against the oracle (1e-7 A, the FP64 tracking bound) for ion
    counts that put the last particle on, before and after a block's edge."""
    s = load(golden_inputs(), "small", n_mg=1 if n_cl else 0, n_cl=n_cl, n_k=n_k)
    o = Oracle(s.to_dict(), seed=3)
    o.populate_lists()
    e = Engine([s], precision=PREC_FP64)
    e.populate_lists()
    e.step(60)
    e.sync()
    o.step(60)
    st, ost = e.get_state(0), o.get_state()
    assert max(np.abs(st[k] - ost[k]).max() for k in "xyz") < 1e-7
    assert e.counters(0)[2] == o.draws()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,steps", [(PREC_MIXED, 120), (PREC_FP64, 20)])
def test_small_and_full_blocks_agree(precision, steps):
    """96 replicas of the small chain (672 particle blocks: full blocks) against two of them
    alone (blocks of few particles): bit for bit in mixed precision, to 1e-9 A in FP64,
    whose sums run in any order."""
    systems = [load(golden_inputs(), "small", seed=s) for s in (3, 4)]
    many, few = Engine(systems * 48, precision=precision), Engine(systems, precision=precision)
    for e in (many, few):
        e.populate_lists()
        e.step(steps)
        e.sync()
    for r in range(2):
        a, b = many.get_state(r + 94), few.get_state(r)
        for k in STATE_NAMES:
            if precision == PREC_MIXED:
                assert np.array_equal(a[k], b[k]), k
            else:
                assert np.abs(a[k] - b[k]).max() < 1e-9, k
        assert many.counters(r + 94) == few.counters(r)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("box,full", [(60.0, 1), (60.0, 0), (67.0, 1), (99.5, 1), (101.0, 0), (133.5, 1), (200.0, 0)])
def test_search_cells_of_any_grid(box, full, precision):
    """The pair sets (and cells) of grids of one and of 2 x 2 x 2 cells (each neighbour met from both
    sides), 3 and more cells per axis, against the oracle's; pruned lists, which the search
    looks for in fewer cells, against the oracle's pairs within their range."""
    s = load(golden_inputs(), "small", box=box, n_mg=4, n_cl=40, n_k=45)
    sd = s.to_dict()
    o = Oracle(sd, seed=3)
    o.populate_lists()
    e = Engine([s], precision=precision, full_lists=full)
    e.populate_lists()
    c, dims = e.cells(0)
    oc, od = o.cells()
    assert np.array_equal(dims, od) and np.array_equal(c, oc)
    sets = [{tuple(sorted(p)) for p in np.asarray(o.pairs(w)).reshape(-1, 2).tolist()} for w in (0, 1)]
    got = [{tuple(p) for p in e.pairs(0, w).tolist()} for w in (0, 1)]
    assert got[1] == sets[1]
    if full:
        assert got[0] == sets[0]
        return
    # a pair with a sugar or base bead is kept within its contact distance plus the skin
    x, kind, typ, rlj = np.stack([sd[k] for k in "xyz"], 1), sd["kind"], sd["type"], sd["rlj"]
    assert got[0] <= sets[0]
    for i, j in sets[0]:
        dv = x[i] - x[j]
        r = np.sqrt(((dv - box * np.round(dv / box)) ** 2).sum())
        charged = kind[i] not in (1, 2) and kind[j] not in (1, 2)
        reach = 3.0 + (3.2 if max(typ[i], typ[j]) <= 6 else rlj[typ[i] - 1] + rlj[typ[j] - 1])
        if charged or abs(r - reach) > 1e-3:
            assert ((i, j) in got[0]) == (charged or r < reach), (i, j, r)
