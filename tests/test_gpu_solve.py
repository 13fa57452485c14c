"""The one-launch Poisson solve (csrc/hf_solve.cuh) at the sizes where its
partition changes: a finest level that is the coarsest (one dense solve), one
CTA, the row counts around each cluster size, ragged last ranks, 3D rows, and
batches whose instances take different cluster sizes; against the same steps in
64-bit torch (perf/cases.py, exact()).

Tolerances: the plain form at Poisson rtol 1e-13 is held to the suite's plain
bar (1e-10 relative L2), the mixed form at the default rtol to the mixed bar
(1e-6: FP32 stencil weights and convection)."""
import importlib.util
import os

import numpy as np
import pytest

from higflow_b200 import engine
from higflow_b200 import program as hp

pytestmark = pytest.mark.gpu

_spec = importlib.util.spec_from_file_location(
    "perf_cases", os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py"))
cases = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(cases)

SIZES = ["9x9", "12x11", "22x23", "23x23", "32x32", "33x31", "45x45", "46x46", "90x91", "91x91", "260x17", "129x128",
         "9x9x9", "10x11x13", "17x16x17", "9,23,46,91", "32,91,10"]


# beyond one cluster: the level-synchronous loop on the folded operators, alone
# and with instances that are all tail or all dense
LARGE = [("300x299", "plain"), ("470x450", "mixed"), ("300,9,40", "plain"), ("460,33,9", "mixed")]


@pytest.mark.parametrize("sides,precision", [(s, p) for p in ("plain", "mixed") for s in SIZES] + LARGE)
def test_steps_match_64_bit_steps(sides, precision):
    flow = "giesekus" if sides in ("23x23", "91x91", "9,23,46,91", "10x11x13") else "newtonian"
    case = dict(flow=flow, sides=sides, steps=3, precision=precision, scheme="explicit", per_step=False, limits="")
    progs = cases._programs(case)
    prog = progs[0] if len(progs) == 1 else hp.Program.concatenate(progs)
    plain = precision == "plain"
    opts = engine.options(precision=hp.PREC_FP64, rtol=1e-13, atol=1e-300) if plain else engine.options(precision=hp.PREC_MIXED)
    c = engine.Case(prog, opts)
    state = dict(case=c, fields=cases._inputs(case, 7)[1], steps=3, per_step=False, limits=None)
    first = cases.run(state)
    again = cases.run(state)
    want = cases.exact(case, 7)
    for k, w in want.items():
        assert np.array_equal(first[k], again[k]), f"{k}: two runs differ"
        err = np.linalg.norm(first[k] - w) / np.linalg.norm(w)
        assert err < (1e-10 if plain else 1e-6), f"{k}: {err:.2e}"
    c.close()


@pytest.mark.parametrize("sides", ["6x5", "16x17", "23x24", "32x33", "33x32", "65x64", "91x90", "128x129", "9x8x10"])
def test_semi_implicit_steps_match_64_bit_steps(sides):
    """The one-launch velocity systems (csrc/hf_bicg.cuh) around the sizes of
    their 256-row blocks and ranks: systems of fewer rows than a block, one rank,
    ragged last blocks, empty last ranks.  Two steps with both solves' residuals
    at 1e-13: u to 1e-10, p (which follows u through div u* / dt, dt = 0.2 h^2)
    to 1e-7."""
    case = dict(flow="oldroyd", sides=sides, steps=2, precision="plain", scheme="semi_implicit", per_step=False, limits="")
    prog = cases._programs(case)[0]
    c = engine.Case(prog, engine.options(precision=hp.PREC_FP64, rtol=1e-13, atol=1e-300))
    got = cases.run(dict(case=c, fields=cases._inputs(case, 7)[1], steps=2, per_step=False, limits=None))
    for k, w in cases.exact(case, 7).items():
        err = np.linalg.norm(got[k] - w) / np.linalg.norm(w)
        assert err < (1e-7 if k == "p" else 1e-10), f"{k}: {err:.2e}"
    c.close()


# clusters smaller than alone (over 148 * 512 rows in all), and instances that
# run in a cluster alone but in the level-synchronous loop beside a larger one
@pytest.mark.parametrize("sides", ["219,155,64,129,33", "460,33,9"])
def test_instances_alone_and_in_a_batch_that_splits_them_otherwise(sides):
    case = dict(flow="newtonian", sides=sides, steps=3, precision="plain", scheme="explicit", per_step=False, limits="")
    progs = cases._programs(case)
    parts, whole = cases._inputs(case, 7)

    def stepped(prog, fields):
        c = engine.Case(prog, engine.options(precision=hp.PREC_FP64, rtol=1e-13, atol=1e-300))
        for (fid, comp), v in fields.items():
            c.set(fid, comp, v)
        c.step(3)
        return c

    batch = stepped(hp.Program.concatenate(progs), whole)
    for i, prog in enumerate(progs):
        alone = stepped(prog, parts[i])
        for fid, comp in ((hp.FIELD_U, 0), (hp.FIELD_U, 1), (hp.FIELD_P, 0)):
            a = alone.get(fid, comp)
            err = np.linalg.norm(batch.get_instance(fid, comp, i) - a) / np.linalg.norm(a)
            assert err < 1e-10, (i, fid, comp, err)
        alone.close()
    batch.close()
