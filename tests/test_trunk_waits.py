"""Waits of the trunk kernels that run out: whole warps give up together, the
launch ends in bounded time with an error status, and the next call on the
same context gives the same results as before."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stalled_call_and_after(lg, c, call, polls=1 << 14, cluster=False):
    """`call` with one wait that nothing satisfies, then without.  cluster:
    the error status is one of the cluster trunk's."""
    good = call()
    c.inject_stall(0, polls)
    t0 = time.perf_counter()
    with pytest.raises(lg.LeelaGPUError) as e:
        call()
    elapsed = time.perf_counter() - t0
    assert e.value.code == -5, str(e.value)  # LG_ERR_DEVICE
    assert elapsed < 20.0
    assert not cluster or 140 < int(str(e.value).split()[-1]) < 150, str(e.value)
    assert np.array_equal(call(), good)
    print(f"stalled call returned after {elapsed * 1e3:.1f} ms: {e.value}")


# 32-channel items on few and on most SMs, 64-channel items
@pytest.mark.parametrize("B", [1, 5, 40])
def test_split_trunk_wait_runs_out(gpu_lib, weights, positions, B):
    lg = gpu_lib
    pp, pv = positions["planes_p"][:B], positions["planes_v"][:B]
    with lg.Context(policy=lg.NetDesc.reference_policy(weights["ref_p"][1]),
                    value=lg.NetDesc.reference_value(weights["ref_v"][1]), max_batch=40) as c:
        c.set_tuning(B, 3, 0)
        _stalled_call_and_after(lg, c, lambda: c.policy(pp))
        _stalled_call_and_after(lg, c, lambda: c.value(pv))


# two layers (the far CTAs of the cluster finish) and eleven (all give up), a
# board alone and all that run side by side
@pytest.mark.parametrize("n3x3", [2, 11])
@pytest.mark.parametrize("B", [1, 36])
def test_cluster_trunk_wait_runs_out(gpu_lib, oracle_mod, positions, n3x3, B):
    lg, O = gpu_lib, oracle_mod
    net = dict(c_in=24, width1=128, width=128, n3x3=n3x3, head_k=1, act=O.RELU, act_head=0)
    pol = O.he_weights(O.make_net(dict(net, value_head=0, fc_hidden=0, value_map=0)), 3)
    pp = positions["planes_p"][:B, :24]
    with lg.Context(policy=lg.NetDesc(pol, 24, 128, 128, n3x3, 1, lg.LG_ACT_RELU, 0, 0, precision="bf16"),
                    max_batch=64) as c:
        c.set_tuning(B, 3, 0)
        _stalled_call_and_after(lg, c, lambda: c.policy(pp), cluster=True)


# 128- and 256-row items, the first layer inside the launch and before it; 64-row
# items (batches of this size run in clusters with choice 3)
@pytest.mark.parametrize("B,choice", [(24, 2), (40, 3), (97, 2), (256, 3)])
def test_persistent_trunk_wait_runs_out(gpu_lib, weights, positions, B, choice):
    lg = gpu_lib
    pv = positions["planes_v"][:B, :24]
    with lg.Context(value=lg.NetDesc.config1_value(weights["cfg_v"][1], "fp16"), max_batch=256) as c:
        c.set_tuning(B, choice, 0)
        _stalled_call_and_after(lg, c, lambda: c.value(pv))
