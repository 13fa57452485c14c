"""A device without room for the one-launch solves' clusters (a partition whose
GPCs offer too few SMs): the case is created and runs on the kernels without
clusters.

The device's answer is replaced on the host: a child process preloads a library
whose hf_clusters_that_fit (csrc/hf_engine.cu) always says 0, and saves its
fields.  Tolerances: explicit velocities run the launch loop instead, which
follows other roundings, so each is held to 64-bit steps at the suite's bars
(plain 1e-10 at Poisson rtol 1e-13, mixed 1e-6).  The velocity systems of the
semi-implicit forms are documented to keep their bits between the one launch
and the separate kernels, and the rest of those steps is the same code: 0."""
import importlib.util
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from higflow_b200 import engine
from higflow_b200 import program as hp

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

_spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(REPO, "perf", "cases.py"))
cases = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(cases)

EXPLICIT = [("9x9", "plain"), ("33x31", "plain"), ("33x31", "mixed"), ("9x10x9", "plain"), ("9,40,20", "mixed")]
BOXES = ["6x5", "33x32", "96x96", "128x129", "180x180", "9x8x10"]
RESIDUALS = ["33x31", "129x128", "240x200", "17x16x17"]
GOLDEN = ["sie2d_cubista", "cn2d_cubista", "bdf2_cav2d", "bdf2_cav3d", "bdf2_oldroyd_log", "cn2d_oldroyd_log",
          "sie2d_oldroyd_log", "amr2d_sie_oldroyd"]


def _box(sides, precision="plain", scheme="explicit"):
    return dict(flow="newtonian" if scheme == "explicit" else "oldroyd", sides=sides, steps=2, precision=precision,
                scheme=scheme, per_step=False, limits="")


def _run(case):
    progs = cases._programs(case)
    prog = progs[0] if len(progs) == 1 else hp.Program.concatenate(progs)
    opts = (engine.options(precision=hp.PREC_MIXED) if case["precision"] == "mixed"
            else engine.options(rtol=1e-13 if case["scheme"] == "explicit" else 1e-10, atol=1e-300))
    c = engine.Case(prog, opts)
    out = cases.run(dict(case=c, fields=cases._inputs(case, 7)[1], steps=case["steps"], per_step=False, limits=None))
    out["loop"], out["launches"] = c.launch_counts()[1], c.stats().kernel_launches
    c.close()
    return out


def _residual_run(sides):
    """One step at Poisson rtol 1e-15: (dp, u*)."""
    case = _box(sides)
    c = engine.Case(cases._programs(case)[0], engine.options(rtol=1e-15, atol=1e-300))
    for k, v in cases._inputs(case, 7)[1].items():
        c.set(*k, v)
    c.step(1)
    out = c.get(hp.FIELD_DP), [c.get(hp.FIELD_USTAR, d) for d in range(c.prog.dim)]
    c.close()
    return out


def _true_residual(sides, dp, us):
    """||b - A dp|| / ||b|| over the rows beside the pinned one, A dp in extended
    precision."""
    case = _box(sides)
    prog, shape = cases._programs(case)[0], cases._shapes(case)[0]
    ex = cases._Exact(prog, shape, "cpu")
    u = [torch.as_tensor(x) for x in us]
    b = sum(ex.q(ex.ds[2 * d + 1], u[d]) - ex.q(ex.ds[2 * d], u[d]) for d in range(prog.dim)).numpy() / ex.h / prog.par["dt"]
    row = np.repeat(np.arange(prog.ncell), np.diff(prog.p_ptr))
    r = b.astype(np.longdouble)
    np.subtract.at(r, row, np.asarray(prog.p_val).astype(np.longdouble) * dp.astype(np.longdouble)[prog.p_col])
    r[prog.pin_row] = 0
    return float(np.sqrt((r * r).sum()) / np.linalg.norm(b))


def _run_golden(name):
    from tests.helpers import field_keys, load_golden, load_init
    prog, data = load_golden(name)
    c = engine.Case(prog, engine.options(rtol=1e-12, atol=1e-300))
    load_init(c, prog, data)
    c.step(3)
    out = {k: c.get(fid, comp) for k, fid, comp in field_keys(prog)}
    out["launches"] = c.stats().kernel_launches
    c.close()
    return out


def _same_bits(got, want, prefix):
    assert want[prefix + "launches"] > got.pop("launches")   # the velocity systems' separate kernels ran there
    for k in got:
        assert np.array_equal(got[k], want[prefix + k]), k


@pytest.fixture(scope="module")
def without_clusters(tmp_path_factory):
    d = tmp_path_factory.mktemp("no_clusters")
    src, lib, out = d / "none.c", d / "none.so", d / "fields.npz"
    src.write_text("int hf_clusters_that_fit(const void *k, const void *c) { (void)k; (void)c; return 0; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=REPO)
    subprocess.run([sys.executable, os.path.abspath(__file__), str(out)], check=True, env=env, cwd=REPO, timeout=600)
    return np.load(out)


@pytest.mark.parametrize("sides,precision", EXPLICIT)
def test_explicit_steps_run_on_the_launch_loop(without_clusters, sides, precision):
    key = f"{sides}/{precision}/"
    assert without_clusters[key + "loop"] > 0
    case = _box(sides, precision)
    assert _run(case)["loop"] == 0        # here, with clusters: the one launch
    for k, want in cases.exact(case, 7).items():
        err = np.linalg.norm(without_clusters[key + k] - want) / np.linalg.norm(want)
        assert err < (1e-10 if precision == "plain" else 1e-6), (k, err)


@pytest.mark.parametrize("sides", RESIDUALS)
def test_the_one_launch_solve_attains_the_loops_residual(without_clusters, sides):
    """The one-launch solve carries q = A z + beta q where the loop multiplies A p
    anew.  Plain solves driven to where ||r|| of the recurrence reaches 1e-15:
    what is left of b - A x itself may be 4 times the loop's (the errors of
    earlier products enter q's with weights beta, beta^2, ...: 1 / (1 - beta) of
    the loop's, beta up to 0.7)."""
    dp, us = _residual_run(sides)
    ours = _true_residual(sides, dp, us)
    loops = _true_residual(sides, without_clusters[f"{sides}/residual/dp"],
                           [without_clusters[f"{sides}/residual/u{d}"] for d in range(len(us))])
    assert 0.0 < ours <= 4.0 * loops, (ours, loops)


@pytest.mark.parametrize("sides", BOXES)
def test_semi_implicit_boxes_keep_their_bits(without_clusters, sides):
    _same_bits(_run(_box(sides, scheme="semi_implicit")), without_clusters, f"{sides}/sie/")


@pytest.mark.parametrize("name", GOLDEN)
def test_semi_implicit_schemes_keep_their_bits(without_clusters, name):
    _same_bits(_run_golden(name), without_clusters, f"{name}/")


def _child(out):
    fields = {}
    for sides, precision in EXPLICIT:
        fields.update({f"{sides}/{precision}/{k}": v for k, v in _run(_box(sides, precision)).items()})
    for sides in RESIDUALS:
        dp, us = _residual_run(sides)
        fields.update({f"{sides}/residual/u{d}": v for d, v in enumerate(us)})
        fields[f"{sides}/residual/dp"] = dp
    for sides in BOXES:
        fields.update({f"{sides}/sie/{k}": v for k, v in _run(_box(sides, scheme="semi_implicit")).items()})
    for name in GOLDEN:
        fields.update({f"{name}/{k}": v for k, v in _run_golden(name).items()})
    np.savez(out, **fields)


if __name__ == "__main__":
    _child(sys.argv[1])
