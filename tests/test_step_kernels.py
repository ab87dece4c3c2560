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
from tis_gb300 import PREC_FP64, PREC_MIXED, STATE_NAMES, Engine, System


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


@pytest.mark.parametrize("box", [51.3, 65.0, 200.0, 250.98, 277.5, 350.0, 501.9, 502.0, 511.9, 1000.0, 4096.0])
def test_position_sums_by_integers(box):
    """The integrator's integer forms (axis_fix, axis_value, shift_fix; constants as tis_create
    forms them) of x + s and of x + (x - x_old) against the FP64 operations, over the axis,
    its ends, neighbours of powers of two, tiny, zero and largest shifts, and ties."""
    rng = random.Random(int(10 * box))
    e = math.frexp(1.02 * box)[1]
    lo, M = (1023 + e - 10) << 20, 2 ** 64 - 1
    span = (_bits(1.01 * box) >> 32) - lo

    def fix(x):
        hi = _bits(x) >> 32
        o = (hi - lo) & 0xFFFFFFFF
        return o < span, (((((hi & 0xFFFFF) | 0x100000) << 32) | (_bits(x) & 0xFFFFFFFF)) << (((o >> 20) + 2) & 15)) & M

    def value(v):
        z = 64 - v.bit_length()
        assert 0 <= z <= 9
        w = (v << z) & M
        up = int((w & 0x7FF) + ((w >> 11) & 1) > 0x400)
        return struct.unpack("<d", struct.pack("<Q", (w >> 11) + ((lo + (8 << 20) - (z << 20)) << 32) + up))[0]

    def shift(s):
        hi = _bits(s) >> 32
        a = hi & 0x7FFFFFFF
        if a >= lo:
            return None
        if s == 0.0:
            return 0
        m = ((((hi & 0xFFFFF) | 0x100000) << 32) | (_bits(s) & 0xFFFFFFFF)) << 1
        r = (lo >> 20) - 1 - (a >> 20)
        v = m >> r if r < 64 else 0
        if r >= 64 or v << r != m:
            v |= 1
        return -v if hi >> 31 else v

    least, fast = 2.0 ** (e - 10), [0, 0]
    for k in range(20000):
        x = rng.uniform(0, box) if k % 4 else rng.choice([box, least, 2.0 ** rng.randint(e - 12, e), 1.0099 * box, 0.0, -1.0])
        x = math.nextafter(x, rng.choice([-1e9, 1e9])) if k % 3 == 0 else x
        s = rng.choice([0.0, 5e-324, 1.0, rng.uniform(-1, 1), 2.0 ** -rng.randint(1, 70)]) * rng.choice([-1, 1]) * math.nextafter(least, 0)
        if k % 5 == 0:  # half a unit in the last place of x, and beside it
            s = math.ulp(x) / 2 * rng.choice([1, -1, 1 + 2.0 ** -52, 1 - 2.0 ** -53])
        ok, v = fix(x)
        if ok:
            assert v == int(math.ldexp(x, 64 - e)) and math.ldexp(x, 64 - e) % 4 == 0
        S = shift(s)
        if ok and S is not None and (v + S) & M >= 2 ** 54:
            fast[0] += 1
            assert value((v + S) & M) == x + s, (x, s)
        o = x - s
        ok2, w = fix(o)
        d = v - w
        if ok and ok2 and -2 ** 54 <= d < 2 ** 54 and (v + d) & M >= 2 ** 54:
            fast[1] += 1
            assert value((v + d) & M) == x + (x - o) == 2.0 * x - o, (x, o)
            a = (d >> 24) * 2.0 ** (e - 40)
            assert abs(a - (x - o)) <= 2.0 ** (e - 40)
    assert min(fast) > 10000


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


@pytest.mark.parametrize("c0", [0, 1, 2, 3, 5046, 2 ** 32 - 2, 2 ** 32 + 3])
@pytest.mark.parametrize("pairs", [1500, 1564])
def test_noise_pairs_of_philox_blocks(pairs, c0):
    """noise_block's split: over threads 0 .. pairs / 2 every pair k is formed once, from draws
    c0 + 2 k and c0 + 2 k + 1, wherever in a block of four the first draw lies."""
    got = {}
    for j in range(pairs // 2 + 1):
        b = (c0 >> 2) + j
        v = [4 * b, 4 * b + 1, 4 * b + 2, 4 * b + 3]
        if c0 & 1:
            v = v[1:] + [4 * b + 4]
        k = 2 * j - ((c0 >> 1) & 1)
        for i in range(2):
            if 0 <= k + i < pairs:
                assert k + i not in got
                got[k + i] = (v[2 * i], v[2 * i + 1])
    assert got == {k: (c0 + 2 * k, c0 + 2 * k + 1) for k in range(pairs)}


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
def test_forces_of_one_replica_among_others(precision):
    """Force terms and ion counts of replicas of different sizes in one handle, read in turn,
    against each replica alone: the results' pinned and device staging holds the largest."""
    systems = [load(golden_inputs(), "small", seed=3, n_mg=1 if n else 0, n_cl=n, n_k=n) for n in (27, 0, 261, 28)]
    many, ones = Engine(systems, precision=precision), [Engine([s], precision=precision) for s in systems]
    for r, one in enumerate(ones):
        for mask in (31, 2):
            f, en = many.forces(r, mask)
            # a call evaluates every replica of its handle and takes its Monte Carlo draws
            g, eg = [e.forces(0, mask) for e in ones][r]
            if precision == PREC_MIXED:
                assert np.array_equal(f, g)
            assert np.abs(f - g).max() <= 1e-9 * np.abs(g).max()  # FP64 sums run in any order
            assert all(abs(en[k] - eg[k]) <= 1e-9 * max(1.0, abs(eg[k])) for k in en), mask
        a, b = many.ion_counts(r, 5, 10.0), one.ion_counts(0, 5, 10.0)
        assert np.array_equal(a[0], b[0]) and a[1] == b[1]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("copies", [5, 6, 8])
def test_monte_carlo_draws_around_the_spare_gaussians(copies, precision):
    """Steps whose Monte Carlo draws fewer and more numbers than the Gaussians made beside it
    leave room for (128): every H-bond candidate several times over and valences of one.  Draw
    counts against the oracle's; states against its (FP64, 1e-7 A) or the drop-in loop's, which
    draws its Gaussians after the Monte Carlo (bit for bit)."""
    sd = load(golden_inputs(), "small").to_dict()
    n, off, co, ci = len(sd["hb_E"]), sd["hb_atom_off"], sd["hba_cand_off"], sd["hba_cand_idx"]
    for k in ("hb_E", "hb_dhs", "hb_dode", "hb_idx", "hb_native", "hb_atom_idx"):
        sd[k] = np.tile(sd[k], copies)
    sd["hb_atom_off"] = np.concatenate([off[:-1] + k * off[-1] for k in range(copies)] + [[copies * off[-1]]]).astype(np.int32)
    sd["hba_cand_off"] = (copies * co).astype(np.int32)
    sd["hba_cand_idx"] = np.concatenate([ci[co[a]:co[a + 1]] + k * n for a in range(len(co) - 1) for k in range(copies)]).astype(np.int32)
    sd["hba_valence"] = np.minimum(sd["hba_valence"], 1).astype(np.int32)
    s = System.from_arrays(sd)
    o = Oracle(s.to_dict(), seed=3)
    a, b = Engine([s], precision=precision), Engine([s], precision=precision)
    for e in (o, a, b):
        e.populate_lists()
    drawn = []
    for _ in range(20):
        before = o.draws()
        o.step(1)
        drawn.append(o.draws() - before - 3000)
        a.step(1)
        a.sync()
        if precision == PREC_FP64:
            assert a.counters(0)[2] == o.draws()
    assert max(drawn) <= 128 if copies == 5 else max(drawn) > 128
    for _ in range(20):
        b.deterministic_forces()
        b.full_forces()
        b.move_rigid_units()
        b.check_shifts()
    b.sync()
    x, y, z = a.get_state(0), b.get_state(0), o.get_state()
    assert a.counters(0) == b.counters(0)
    for k in STATE_NAMES:
        assert np.array_equal(x[k], y[k]) if precision == PREC_MIXED else np.abs(x[k] - y[k]).max() < 1e-9, k
    if precision == PREC_FP64:
        assert max(np.abs(x[k] - z[k]).max() for k in "xyz") < 1e-7


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 48])
def test_skin_check_in_either_kernel(copies):
    """The drop-in loop, whose integrator ends with the skin check, against steps, whose cell
    kernel begins with it, over list rebuilds: bit for bit in mixed precision."""
    systems = [load(golden_inputs(), "small", seed=s) for s in (3, 4)] * copies
    a, b = Engine(systems, precision=PREC_MIXED), Engine(systems, precision=PREC_MIXED)
    for e in (a, b):
        e.populate_lists()
    a.step(150)
    for _ in range(150):
        b.deterministic_forces()
        b.full_forces()
        b.move_rigid_units()
        b.check_shifts()
    for e in (a, b):
        e.sync()
    assert max(a.counters(r)[1] for r in range(len(systems))) > 1
    for r in (0, len(systems) - 1):
        assert a.counters(r) == b.counters(r)
        x, y = a.get_state(r), b.get_state(r)
        for k in STATE_NAMES:
            assert np.array_equal(x[k], y[k]), k


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


@pytest.mark.gpu
@pytest.mark.parametrize("n,box,sr,lr,offset", [(1, (40.0,) * 3, 5.0, 20.0, 0), (33, (40.0, 61.0, 95.0), 7.0, 20.0, 1),
                                                (700, (70.0, 75.0, 200.0), 15.0, 33.0, 1), (2049, (150.0,) * 3, 15.0, 15.0, 0),
                                                (4000, (120.0, 99.0, 101.5), 10.0, 33.0, 1)])
def test_noalloc_pairs_of_any_grid(n, box, sr, lr, offset):
    """tis_pair_lists_noalloc over grids of one to ten cells per axis, particles on the faces,
    outside the box (wrapped once, or left out and counted), equal radii, capacities that cut
    the output and an output array aligned to four bytes, against all pairs in FP64 numpy."""
    import torch
    from tis_gb300 import api
    rng = np.random.default_rng(n)
    L = np.asarray(box)
    x = rng.uniform(-0.2, 1.2, (n, 3)) * L  # differences within 1.5 box sides: the image rule gives the nearest
    x[rng.random((n, 3)) < 0.02] = 0.0
    if n > 500:
        x[: n // 3] = L / 3 + rng.normal(size=(n // 3, 3)) * 8.0  # a dense cluster
        x[:3] = 3.0 * L  # beyond the single wrap
    kind = rng.integers(0, 6, n).astype(np.int32)
    # separate_in_cells (E:1461-1542): one wrap, then ceil(x / l), which puts x = 0 in no cell
    m = (L / lr).astype(int)
    w = np.where(x < 0, x + L, np.where(x > L, x - L, x))
    cell = np.ceil(w / (L / m))
    inside = ((cell >= 1) & (cell <= m)).all(1)
    i, j = np.triu_indices(n, 1)
    ok = inside[i] & inside[j]
    i, j = i[ok], j[ok]
    d = x[i] - x[j]
    d = np.where(d > 0.5 * L, d - L, d)
    d = np.where(d < -0.5 * L, d + L, d)
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
    charged = (kind != 1) & (kind != 2)
    is_sr = r2 <= sr * sr
    want = [np.stack([i[m], j[m]], 1) for m in (is_sr, ~is_sr & (r2 <= lr * lr) & charged[i] & charged[j])]
    xyz = [torch.from_numpy(np.ascontiguousarray(x[:, c])).cuda() for c in range(3)]
    k = torch.from_numpy(kind).cuda()
    for cut in (1.0, 0.5):
        caps = [max(1, int(cut * len(w)) + (64 if cut == 1.0 else 0)) for w in want]
        out = [torch.full((2 * c + 3,), -7, dtype=torch.int32, device="cuda") for c in caps]
        counts = torch.full((3,), -1, dtype=torch.int64, device="cuda")
        api.pair_lists_noalloc(*[v.data_ptr() for v in xyz], k.data_ptr(), n, L, sr, lr, out[0].data_ptr() + 4 * offset, caps[0],
                               out[1].data_ptr() + 4 * offset, caps[1], counts.data_ptr(), torch.cuda.current_stream().cuda_stream)
        c = counts.cpu().numpy()
        assert c.tolist() == [len(want[0]), len(want[1]), int((~inside).sum())]
        for w, o, cap in zip(want, out, caps):
            o = o.cpu().numpy()
            m = min(cap, len(w))
            got = {tuple(p) for p in o[offset: offset + 2 * m].reshape(-1, 2).tolist()}
            assert len(got) == m and got <= {tuple(p) for p in w.tolist()}
            assert (o[:offset] == -7).all() and (o[offset + 2 * m:] == -7).all()


@pytest.mark.gpu
def test_gradients_of_small_and_full_blocks_agree():
    """dU/dtheta and a trajectory gradient of replicas on full blocks (a handle of 96) against
    the same replicas alone, on blocks of few particles: FP64 sums in another order."""
    systems = [load(golden_inputs(), "small", seed=s) for s in (3, 4)]
    many, few = (Engine(s, precision=PREC_MIXED, groups=1) for s in (systems * 48, systems))
    for e in (many, few):
        e.populate_lists()
        e.step(200)
        e.sync()
    a, b = many.param_grad(), few.param_grad()
    assert np.abs(a[:2] - b).max() <= 1e-10 * np.abs(b).max() and np.array_equal(a[94:] != 0, b != 0)
    n = sum(few.n)
    w = np.random.default_rng(5).normal(size=n)
    ga, da = many.traj_grad(6, 4, {"x": np.tile(w, 48)}, want_state=True)
    gb, db = few.traj_grad(6, 4, {"x": w}, want_state=True)
    assert np.abs(ga[:2] - gb).max() <= 1e-9 * np.abs(gb).max()
    for k in STATE_NAMES:
        assert np.abs(da[k][:n] - db[k]).max() <= 1e-9 * max(1.0, np.abs(db[k]).max()), k


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["same", "turned", "half_turn", "noisy", "unrelated", "mirrored", "three", "line"])
def test_fit_of_any_frame(kind):
    """The least-squares fit's rmsd against a singular value decomposition's, for frames that
    fit exactly, turned by any angle and by pi (a vanishing quaternion component), with noise,
    unrelated, mirrored, of three beads, and on a line (a double eigenvalue)."""
    rng = np.random.default_rng(len(kind))
    s = load(golden_inputs(), "small")
    e = Engine([s], precision=PREC_MIXED)
    st = e.get_state(0)
    beads = np.arange(0, 3 if kind == "three" else 60, 1).astype(np.int32)
    if kind == "line":
        t = np.linspace(-30, 30, len(beads))
        for k, u in zip("xyz", (0.6, 0.0, 0.8)):
            st[k][beads] = 100.0 + u * t
            st["o" + k][beads] = st[k][beads]
        e.set_state(0, st)
    x = np.stack([st[k][beads] for k in "xyz"], 1)
    q = {"half_turn": np.array([0.0, 0.6, 0.0, 0.8])}.get(kind, rng.normal(size=4))
    q /= np.linalg.norm(q)
    w, v = q[0], q[1:]
    K = np.array([[0, -v[2], v[1]], [v[2], 0, -v[0]], [-v[1], v[0], 0]])
    R = np.eye(3) if kind == "same" else np.eye(3) + 2 * w * K + 2 * K @ K
    ref = (x - x.mean(0)) @ R.T + rng.normal(size=3) * 40
    if kind == "noisy":
        ref += rng.normal(size=ref.shape) * 3.0
    elif kind == "unrelated":
        ref = rng.normal(size=ref.shape) * 20.0
    elif kind == "mirrored":
        ref[:, 0] *= -1.0
    g = e.density(0, 5, (0.0, 0.0, 0.0), 5.0, (40, 40, 40), beads, ref)
    g.add()
    rmsd = g.get()[2]
    a, b = x - x.mean(0), ref - ref.mean(0)
    U, sv, Vt = np.linalg.svd(a.T @ b)
    sv[2] *= np.sign(np.linalg.det(Vt.T @ U.T)) or 1.0
    want = np.sqrt(max(0.0, (a * a).sum() + (b * b).sum() - 2 * sv.sum()) / len(beads))
    # the reference value cancels its sums: good to sqrt(2^-52) of the spread
    assert abs(rmsd - want) < 3e-8 * np.sqrt((a * a).sum() / len(beads)) + 1e-9 * want, (rmsd, want)
