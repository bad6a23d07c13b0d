"""A copy of one batch member's records that never completes (hc_batch_inject_stalled_copy): every
member that it spoils is marked, the others' results are those of an undisturbed batch bit for bit,
and the batch steps on once the hook is cleared."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300._capi import HC_ERR_TIMEOUT, HCError, StepStats
from hyperboliconvergence_gb300.batch import Batch

pytestmark = pytest.mark.gpu
N = 64


def make():
    rng = np.random.default_rng(12)
    insts = [cases.gaussian_sum(48, 60, rng)[:4] for _ in range(N)]
    b = Batch(insts, flux="slau", limiter="vanalbada", precision="fp32", species=(1.4, 287.058, 0.3))
    b.set_schedule("8x32", ctas_per_sm=1)  # fewer warps than strip runs: a warp serves several members
    return b, insts


def step(b, mode):
    b.step_async(1, mode)
    st = (StepStats * N)()
    code = b.lib.hc_batch_sync(b.h, st)
    return code, [s.status for s in st], [b.get_state(k) for k in range(N)]


@pytest.mark.parametrize("mode", ["persistent", "per_instance"])
def test_stalled_member(mode):
    b, insts = make()
    code, status, good = step(b, mode)
    assert code == 0 and not any(status)
    b, _ = make()
    b.inject_stalled_copy(0)
    code, status, states = step(b, mode)
    assert code != 0 and status[0] != 0
    for k in range(N):
        if status[k] == 0:
            assert np.array_equal(states[k], good[k]), k
    spoiled = sum(s != 0 for s in status)
    assert 1 < spoiled < N if mode == "persistent" else spoiled == 1
    b.inject_stalled_copy(-1)
    for k, inst in enumerate(insts):
        b.set_state(k, inst[3])
    code, status, states = step(b, mode)
    assert code == 0 and not any(status)
    assert all(np.array_equal(x, y) for x, y in zip(states, good))


def test_timeout_is_reported_as_such():
    b, _ = make()
    b.inject_stalled_copy(3)
    code, status, _ = step(b, "per_instance")
    assert code == HC_ERR_TIMEOUT
    assert [s for s in status if s] == [HC_ERR_TIMEOUT] and status[3] == HC_ERR_TIMEOUT
    b.step_async(1, "per_instance")
    with pytest.raises(HCError) as err:
        b.sync()
    assert err.value.code == HC_ERR_TIMEOUT
