"""Which kernels a case's Poisson solve runs on (csrc/hf_solve.cuh in one launch,
or the launch loop on the folded operators), and both on forms of the operator
beside 5- and 7-entry rows in row-major order.

hf_case_launch_counts reports the kernels of one loop body: 0 for the one-launch
solve.  Tolerances as in test_gpu_solve.py: plain at Poisson rtol 1e-13 1e-10
relative L2, mixed 1e-6."""
import copy

import numpy as np
import pytest

from higflow_b200 import engine
from higflow_b200 import program as hp
from tests.test_gpu_solve import LARGE, SIZES, cases

pytestmark = pytest.mark.gpu


def _options(precision, **kw):
    if precision == "plain":
        return engine.options(precision=hp.PREC_FP64, rtol=1e-13, atol=1e-300, **kw)
    return engine.options(precision=hp.PREC_MIXED, **kw)


def _case(sides, precision="plain", flow="newtonian", steps=2):
    return dict(flow=flow, sides=sides, steps=steps, precision=precision, scheme="explicit", per_step=False, limits="")


def _program(case):
    progs = cases._programs(case)
    return progs[0] if len(progs) == 1 else hp.Program.concatenate(progs)


def _run(prog, opts, fields, steps):
    c = engine.Case(prog, opts)
    out = cases.run(dict(case=c, fields=fields, steps=steps, per_step=False, limits=None))
    loop = c.launch_counts()[1]
    c.close()
    return out, loop


@pytest.mark.parametrize("sides,precision", [(s, p) for p in ("plain", "mixed") for s in SIZES] + LARGE)
def test_the_sizes_tested_take_the_route_they_stand_for(sides, precision):
    c = engine.Case(_program(_case(sides)), _options(precision))
    c.step(1)
    assert (c.launch_counts()[1] > 0) == ((sides, precision) in LARGE)
    c.close()


# beside an instance beyond a cluster: instances whose whole V-cycle is the tail
# kernel, finest level included (129 to 1,024 rows)
@pytest.mark.parametrize("sides,precision", [("300,20,31", "plain"), ("460,25,9,12", "mixed")])
def test_the_loops_tail_from_the_finest_level(sides, precision):
    case = _case(sides, precision, steps=3)
    got, loop = _run(_program(case), _options(precision), cases._inputs(case, 7)[1], 3)
    assert loop > 0
    for k, want in cases.exact(case, 7).items():
        err = np.linalg.norm(got[k] - want) / np.linalg.norm(want)
        assert err < (1e-10 if precision == "plain" else 1e-6), (k, err)


# the largest velocity systems of the one launch, and systems beyond it
@pytest.mark.parametrize("sides", ["180x180", "210x210"])
def test_semi_implicit_steps_around_the_cluster_limit(sides):
    """u to 1e-10, p (which follows u through div u* / dt, dt = 0.2 h^2) to 1e-7."""
    case = dict(_case(sides, flow="oldroyd"), scheme="semi_implicit")
    got, _ = _run(_program(case), _options("plain"), cases._inputs(case, 7)[1], 2)
    for k, want in cases.exact(case, 7).items():
        err = np.linalg.norm(got[k] - want) / np.linalg.norm(want)
        assert err < (1e-7 if k == "p" else 1e-10), (k, err)


def _compact(prog, shape):
    """The program with the full neighbour stencil (9 entries in 2D, 27 in 3D) in
    its Poisson rows: weights falling with the distance, zero row sums,
    symmetric."""
    prog = copy.copy(prog)   # (cases shares its programs)
    n, D, h2 = prog.ncell, len(shape), float(prog.delta[0, 0]) ** 2
    idx = np.stack([g.ravel() for g in np.meshgrid(*[np.arange(m) for m in shape], indexing="ij")], 1)
    cols, vals = [], []
    for move in np.ndindex(*[3] * D):
        move = np.array(move) - 1
        far = int(np.abs(move).sum())
        if far == 0:
            continue
        J = idx + move
        ok = ((J >= 0) & (J < np.array(shape))).all(1)
        cols.append(np.where(ok, np.ravel_multi_index(tuple(np.where(ok[:, None], J, 0).T), shape), -1))
        vals.append(np.where(ok, 4.0 ** (1 - far) / h2, 0.0))
    cols, vals = np.stack(cols, 1), np.stack(vals, 1)
    cols = np.concatenate([np.arange(n)[:, None], cols], 1)
    vals = np.concatenate([-vals.sum(1)[:, None], vals], 1)
    keep = cols >= 0
    keep[prog.pin_row] = False
    prog.p_ptr = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int64)
    prog.p_col, prog.p_val = cols[keep].astype(np.int32), vals[keep]
    return prog


# 512 and 1024 threads a CTA, both forms; one finest level that is the coarsest
@pytest.mark.parametrize("sides", ["9x9", "33x31", "170x160", "9x10x11"])
@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_rows_of_more_entries_than_a_uniform_grids(sides, precision):
    """Against Jacobi-preconditioned CG, which no hierarchy or template of the
    one-launch solve enters."""
    case = _case(sides)
    prog = _compact(_program(case), cases._shapes(case)[0])
    fields = cases._inputs(case, 7)[1]
    want, _ = _run(prog, _options("plain", precond=hp.PRECOND_JACOBI), fields, 2)
    got, loop = _run(prog, _options(precision), fields, 2)
    assert loop == 0
    for k in want:
        err = np.linalg.norm(got[k] - want[k]) / np.linalg.norm(want[k])
        assert err < (1e-10 if precision == "plain" else 1e-6), (k, err)


def _renumbered(prog, new):
    """The (Newtonian) program with cell i as cell new[i]."""
    prog = copy.copy(prog)
    old = np.argsort(new)
    slots = []
    for s in prog.vel_slots:
        s = s.copy()
        for k in (hp.V_PR, hp.V_PL):
            assert (s[k] >= 0).all()
            s[k] = new[s[k]]
        slots.append(s)
    prog.vel_slots = slots
    prog.div_slots = np.ascontiguousarray(np.asarray(prog.div_slots)[:, old])
    ptr = np.asarray(prog.p_ptr)
    at = [np.arange(ptr[i], ptr[i + 1]) for i in old]
    prog.p_ptr = np.concatenate([[0], np.cumsum([len(a) for a in at])]).astype(np.int64)
    at = np.concatenate(at)
    prog.p_col, prog.p_val = new[np.asarray(prog.p_col)[at]].astype(np.int32), np.asarray(prog.p_val)[at]
    prog.pin_row = int(new[prog.pin_row])
    return prog


# every rank reaching every other's rows; many cells in random order have too many
# row templates for shared memory and run the loop
@pytest.mark.parametrize("order", ["reversed", "random"])
@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("sides", ["9x9", "20x20", "45x46", "9x9x9"])
def test_cells_in_another_order(sides, precision, order):
    case = _case(sides, precision)
    want = cases.exact(case, 7)
    prog = _program(case)
    new = (np.arange(prog.ncell)[::-1].copy() if order == "reversed"
           else np.random.default_rng(5).permutation(prog.ncell))
    fields = dict(cases._inputs(case, 7)[1])
    for k in ((hp.FIELD_P, 0), (hp.FIELD_DP, 0)):
        fields[k] = fields[k][np.argsort(new)]
    got, loop = _run(_renumbered(prog, new), _options(precision), fields, 2)
    assert loop == 0 or (order == "random" and prog.ncell > 400)
    got["p"] = got["p"][new]
    for k in want:
        err = np.linalg.norm(got[k] - want[k]) / np.linalg.norm(want[k])
        assert err < (1e-10 if precision == "plain" else 1e-6), (k, err)


@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_steps_after_a_case_that_left_nan_in_shared_memory(precision):
    """The padding of a coarse level's slices multiplies element 0 of the
    cluster's shared memory by zero: that element has to be set first, whatever
    the kernel before left there.  A batch of NaN instances covers every SM,
    then one without steps as ever."""
    case = _case("33x33", precision)
    prog = _program(case)
    many = hp.Program.concatenate([prog] * 300)
    bad = engine.Case(many, _options(precision))
    bad.set(hp.FIELD_U, 0, np.full(300 * prog.nfacet[0], np.nan))
    with pytest.raises(engine.EngineError) as e:
        bad.step(1)
    assert e.value.code == -4
    got, loop = _run(prog, _options(precision), cases._inputs(case, 7)[1], 2)
    bad.close()
    assert loop == 0
    for k, want in cases.exact(case, 7).items():
        err = np.linalg.norm(got[k] - want) / np.linalg.norm(want)
        assert err < (1e-10 if precision == "plain" else 1e-6), (k, err)
