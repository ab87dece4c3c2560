"""What the step's kernels and the calls around them hold to in every form they take: which
terms a list entry has, the order of FP64 sums, the memory a call leaves behind."""
import numpy as np
import pytest

from oracle_bridge import Oracle
from systems import golden_inputs, load, rel_err
from tis_gb300 import PREC_FP64, PREC_MIXED, STATE_NAMES, TERM_LR, TERM_SR, Engine


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(PREC_MIXED, 1e-5), (PREC_FP64, 1e-10)])
def test_lr_entries_inside_the_contact_distance(precision, tol):
    """An SR list radius (4 A) below the contact distances of phosphate and K+ (4.76 A): the pairs
    between the two are LR entries and feel Coulomb alone (E:1851-1907).  The LR term against the
    oracle's (the per-term bounds), one step against the oracle's in FP64 (1e-7 A) and against the
    persistent kernel's in mixed precision (bit for bit)."""
    s = load(golden_inputs(), "small")
    e = Engine([s], precision=PREC_FP64)
    e.populate_lists()
    e.step(300)
    e.sync()
    st = e.get_state(0)
    o = Oracle(s.to_dict(), seed=3, sr=3.0, skin=1.0)
    o.set_state(st)
    o.populate_lists()
    sd = s.to_dict()
    i, j = np.asarray(o.pairs(1)).reshape(-1, 2).T
    dv = np.stack([st[k][i] - st[k][j] for k in "xyz"], 1)
    r = np.sqrt(((dv - 200.0 * np.round(dv / 200.0)) ** 2).sum(1))
    typ, rlj = sd["type"], sd["rlj"]
    assert (r < np.where(np.maximum(typ[i], typ[j]) <= 6, 3.2, rlj[typ[i] - 1] + rlj[typ[j] - 1])).sum() > 0
    ref = o.terms()
    a = Engine([s], precision=precision, sr=3.0, skin=1.0)
    a.set_state(0, st)
    a.populate_lists()
    f, en = a.forces(0, TERM_LR)
    assert rel_err(f, ref["F_lr"]) < tol and en["E_lj"] == 0.0
    assert en["E_coul_lr"] == pytest.approx(ref["E_coul_lr"], rel=tol)
    a.step(1)
    a.sync()
    x = a.get_state(0)
    if precision == PREC_FP64:
        o.step(1)
        y = o.get_state()
        assert max(np.abs(x[k] - y[k]).max() for k in "xyz") < 1e-7
        return
    b = Engine([s], precision=precision, sr=3.0, skin=1.0, fused_ctas=1)
    b.set_state(0, st)
    b.populate_lists()
    b.step(1)
    b.sync()
    y = b.get_state(0)
    for k in STATE_NAMES:
        assert np.array_equal(x[k], y[k]), k


@pytest.mark.gpu
def test_fp64_pair_forces_keep_an_order():
    """FP64 SR and held LR forces are the same bits on every evaluation, and in a handle large
    enough for full blocks: each particle's entries are summed in an order its list alone sets.
    Also against the oracle's terms (1e-10, the FP64 bound)."""
    s = load(golden_inputs(), "small")
    e, many = Engine([s], precision=PREC_FP64), Engine([s] * 96, precision=PREC_FP64)
    e.populate_lists()
    e.step(300)
    e.sync()
    st = e.get_state(0)
    e.set_state(0, st)
    e.populate_lists()
    o = Oracle(s.to_dict(), seed=3)
    o.set_state(st)
    o.populate_lists()
    ref = o.terms()
    for term, name in ((TERM_SR, "F_sr"), (TERM_LR, "F_lr")):
        f = e.forces(0, term)[0]
        assert rel_err(f, ref[name]) < 1e-10
        for _ in range(20):
            assert np.array_equal(f, e.forces(0, term)[0])
    # ions feel SR and LR forces alone: one thread's sum of each, in both launch shapes
    many.set_states({k: np.tile(st[k], 96) for k in STATE_NAMES})
    many.populate_lists()
    ions = slice(3 * int(s["n_rna"][0]), None)
    for h in (e, many):
        h.deterministic_forces()
    f = e.current_forces(0)[ions]
    for r in (0, 41, 95):
        assert np.array_equal(f, many.current_forces(r)[ions])


@pytest.mark.gpu
def test_gradient_memory_of_a_handle_of_groups():
    """What a trajectory gradient leaves reserved for the next call does not grow with the number of
    replica groups, which take it in turn: six groups of one replica hold less than twice what
    one replica alone does (and 64 MiB, the allocator's rounding); closing the handle gives it back."""
    import torch
    s = load(golden_inputs(), "small")

    def held(replicas):
        e = Engine([s] * replicas, precision=PREC_MIXED, groups=replicas)
        e.populate_lists()
        e.sync()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for _ in range(2):
            e.traj_grad(80, 40, {"x": np.ones(sum(e.n))})
        torch.cuda.synchronize()
        left = free - torch.cuda.mem_get_info()[0]
        e.close()
        return left, torch.cuda.mem_get_info()[0] - free

    held(1)  # modules loaded
    one, six = held(1), held(6)
    assert six[0] < 2 * one[0] + (64 << 20), (one, six)
    assert min(one[1], six[1]) >= 0  # the handle's own memory came back too


@pytest.mark.gpu
def test_gradients_beyond_the_memory_kept():
    """100 steps of 64 replicas in one segment (over the 4 GiB that a handle keeps between calls) and
    in segments of 20 (below) give the same gradients: 1e-8, where the order of FP64 sums leaves
    about 1e-14 after 40 steps.  Of the former call nothing stays behind but the rounding of allocations."""
    import torch
    s = load(golden_inputs(), "small")

    def gradients(every):
        e = Engine([s] * 64, precision=PREC_MIXED, groups=1)
        st = e.get_states()
        seed = {"x": np.random.default_rng(1).normal(size=sum(e.n))}
        e.traj_grad(3, 3, seed)  # streams, events and the pool are made, the lists have grown
        e.set_states(st)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        g, d0 = e.traj_grad(100, every, seed, want_state=True)
        torch.cuda.synchronize()
        left = free - torch.cuda.mem_get_info()[0]
        e.close()
        return g, d0, left

    (g, d0, left), (g2, d2, _) = gradients(100), gradients(20)
    assert left <= 64 << 20
    assert rel_err(g, g2) < 1e-8
    for k in d0:
        assert rel_err(d0[k], d2[k]) < 1e-8, k
