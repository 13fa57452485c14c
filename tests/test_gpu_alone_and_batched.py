"""A case alone, in a batch that splits it otherwise, and in a served mix.

A batch's row count sets the clusters of its instances, and an instance beside
one too large for a cluster runs the launch loop, so the results agree to the
Poisson solve and not to the bit.  What that allows, per field: two solves of one
system to ||r|| <= rtol ||b|| differ by at most 2 rtol ||b|| / lambda_min in the
increment of p, that is 2 rtol kappa of it, kappa = 8 n^2 / pi^2 on n cells a side
(lambda_max = 8 / h^2, lambda_min = pi^2); and in u by dt times the gradient of
that difference, 2 rtol ||div u*|| / pi <= 2 rtol sqrt(8) n / pi of u.  Both for
every step taken (the steps damp differences of u: explicit, below the stability
bound), the plain form at rtol 1e-13 held to the suite's 1e-10 besides."""
import time

import numpy as np
import pytest

from higflow_b200 import engine, serve
from higflow_b200 import program as hp
from tests.test_gpu_solve import cases

pytestmark = pytest.mark.gpu
FIELDS = ((hp.FIELD_U, 0), (hp.FIELD_U, 1), (hp.FIELD_P, 0))


def _bound(key, n, rtol, steps):
    return 2.0 * rtol * steps * (8.0 * n * n / np.pi ** 2 if key[0] == hp.FIELD_P else np.sqrt(8.0) * n / np.pi)


def _boxes(sides, steps):
    case = dict(flow="newtonian", sides=sides, steps=steps, precision="plain", scheme="explicit", per_step=False, limits="")
    return cases._programs(case), cases._shapes(case), cases._inputs(case, 7)


def _alone(prog, fields, steps, **kw):
    c = engine.Case(prog, engine.options(**kw))
    for k, v in fields.items():
        c.set(*k, v)
    c.step(steps)
    out = {k: c.get(*k) for k in FIELDS}
    c.close()
    return out


# clusters smaller than alone, and instances in the loop beside a larger one
@pytest.mark.parametrize("sides,precision", [("219,155,64,129,33", hp.PREC_FP64), ("219,155,64,129,33", hp.PREC_MIXED),
                                             ("300,33,9", hp.PREC_FP64), ("460,33,9", hp.PREC_MIXED)])
def test_batches_at_the_default_tolerance(sides, precision):
    steps, rtol = 3, 1e-10
    progs, shapes, (parts, whole) = _boxes(sides, steps)
    opts = dict(rtol=rtol, atol=1e-300, precision=precision)
    c = engine.Case(hp.Program.concatenate(progs), engine.options(**opts))
    for k, v in whole.items():
        c.set(*k, v)
    c.step(steps)
    for i, prog in enumerate(progs):
        alone = _alone(prog, parts[i], steps, **opts)
        for k in FIELDS:
            err = np.linalg.norm(c.get_instance(*k, i) - alone[k]) / np.linalg.norm(alone[k])
            assert err < _bound(k, shapes[i][0], rtol, steps), (i, k, err)
    c.close()


REQUESTS = ("33,219,64,155,129,40,181", (7, 3, 9, 4, 6, 12, 3))


def test_served_requests_agree_with_their_runs_alone():
    """Requests grouped into cohorts that step as one batch, each frozen at its
    own step count: 1e-10 relative L2 at Poisson rtol 1e-13."""
    sides, counts = REQUESTS
    progs, _, (parts, _) = _boxes(sides, 1)
    opts = dict(rtol=1e-13, atol=1e-300)
    srv = serve.BatchServer(opts=engine.options(**opts), max_cohorts=2, chunk=3)
    ids = []
    for i, prog in enumerate(progs):
        ids.append(srv.submit(prog, counts[i], parts[i]))
        if i == 4:
            time.sleep(0.3)       # the last ones arrive while the first cohort runs or after it
    for i, rid in enumerate(ids):
        assert srv.wait(rid, timeout=300)[0] == 0
        alone = _alone(progs[i], parts[i], counts[i], **opts)
        for k in FIELDS:
            err = np.linalg.norm(srv.get(rid, *k) - alone[k]) / np.linalg.norm(alone[k])
            assert err < 1e-10, (i, k, err)
        srv.release(rid)
    srv.close()


def test_a_served_request_with_a_nan_fails_alone():
    sides, counts = REQUESTS
    progs, _, (parts, _) = _boxes(sides, 1)
    opts = dict(rtol=1e-13, atol=1e-300)
    bad = {k: v.copy() for k, v in parts[1].items()}
    bad[hp.FIELD_U, 0][5] = np.nan
    srv = serve.BatchServer(opts=engine.options(**opts), max_cohorts=1, chunk=2)
    ids = [srv.submit(p, counts[i], bad if i == 1 else parts[i]) for i, p in enumerate(progs)]
    assert [srv.wait(rid, timeout=300)[0] for rid in ids] == [-4 if i == 1 else 0 for i in range(len(ids))]
    for i, rid in enumerate(ids):
        if i == 1:
            continue
        alone = _alone(progs[i], parts[i], counts[i], **opts)
        for k in FIELDS:
            err = np.linalg.norm(srv.get(rid, *k) - alone[k]) / np.linalg.norm(alone[k])
            assert err < 1e-10, (i, k, err)
    srv.close()


def test_requests_as_cases_of_their_own_keep_their_bits():
    """hf_server_*: each request an engine case of its own, so nothing of the mix
    enters its result."""
    sides, counts = REQUESTS
    progs, _, (parts, _) = _boxes(sides, 1)
    srv = engine.Server(max_active=4, chunk_steps=2, setup_threads=2)
    ids = [srv.submit(p, engine.options(), counts[i], parts[i]) for i, p in enumerate(progs)]
    for i, rid in enumerate(ids):
        assert srv.wait(rid)[0] == 0
        alone = _alone(progs[i], parts[i], counts[i])
        for k in FIELDS:
            assert np.array_equal(srv.get(rid, *k), alone[k]), (i, k)
        srv.release(rid)
    srv.close()
