"""Steps queued without waiting (hf_case_step_async): what the calls after them
return and wait for."""
import numpy as np
import pytest
import torch

from higflow_b200 import engine
from higflow_b200 import program as hp
from tests.helpers import load_golden, load_init

pytestmark = pytest.mark.gpu


def _case(**kw):
    prog, data = load_golden("cav2d_cubista")
    case = engine.Case(prog, engine.options(rtol=1e-10, atol=1e-300, **kw))
    load_init(case, prog, data)
    return case, prog


def _state(case):
    s = case.stats()
    return (case.instance_iters().tolist(), case.instance_result(0), case.instance_failures().tolist(), s.total_iters,
            s.last_residual, s.kernel_launches)


@pytest.mark.parametrize("eager", [False, True])
@pytest.mark.parametrize("profile", [False, True])
def test_solver_state_after_queued_steps_is_that_of_the_last_step(profile, eager):
    """The solver's results and counters describe the last step queued, with
    or without phase timing and whether or not the caller synchronises first."""
    case, _ = _case(eager=eager)
    case.profile(profile)
    case.step(2)
    before = _state(case)
    for n in (1, 3):
        case.step(n, sync=False)
        got = _state(case)
        case.synchronize()
        assert got == _state(case)
        assert got[0][0] > before[0][0]
        before = got
    case.close()


def test_failure_of_a_queued_step_is_seen_under_profiling():
    case, prog = _case()
    case.set_step_limits([8])
    case.profile(True)
    case.step(1)
    assert list(case.instance_failures()) == [0]
    u = case.get(hp.FIELD_U, 0)
    u[3] = np.nan
    case.set(hp.FIELD_U, 0, u)
    case.step(1, sync=False)
    assert list(case.instance_failures()) == [-4]
    assert case.instance_result(0)[2] == -4
    with pytest.raises(engine.EngineError) as e:
        case.synchronize()
    assert e.value.code == -4
    case.close()


@pytest.mark.parametrize("call", ["set_timestep", "set_field"])
def test_writing_calls_wait_for_the_steps_queued_before_them(call):
    """hf_case_set_timestep and hf_case_set_field wait for the case's queued
    steps, so that an error of theirs is not left to a later call."""
    case, prog = _case()
    case.step(1)
    u = case.get(hp.FIELD_U, 0)
    case.step(1000, sync=False)
    done = torch.cuda.Event()
    done.record(torch.cuda.ExternalStream(case.stream()))
    assert not done.query()
    if call == "set_timestep":
        case.set_timestep(prog.par["dt"])
    else:
        case.set(hp.FIELD_U, 0, u)
    assert done.query()
    case.close()
