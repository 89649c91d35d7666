"""Host calls hand back the device calls' bits on both sides of the size up
to which a kernel writes the results into pinned memory (8,192 floats)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("B", [1, 22, 23, 45])
def test_host_results_equal_device_results(gpu_lib, weights, positions, prec, B):
    """22 positions' probabilities are the largest in one kernel, 23 the
    smallest by copies; 45 is a chunk of 23 and one of 22."""
    import torch
    lg = gpu_lib
    pp = np.ascontiguousarray(positions["planes_p"][:B, :24])
    pv = np.ascontiguousarray(positions["planes_v"][:B, :24])
    with lg.Context(policy=lg.NetDesc.config1_policy(weights["cfg_p"][1], prec),
                    value=lg.NetDesc.config1_value(weights["cfg_v"][1], prec), max_batch=23) as c:
        dp, dv = torch.from_numpy(pp).cuda(), torch.from_numpy(pv).cuda()
        probs = torch.empty(B, 361, device="cuda")
        logits = torch.empty(B, 361, device="cuda")
        value = torch.empty(B, device="cuda")
        torch.cuda.synchronize()
        c.policy_device(dp.data_ptr(), B, probs.data_ptr(), 0.75, logits_ptr=logits.data_ptr())
        c.value_device(dv.data_ptr(), B, value.data_ptr())
        torch.cuda.synchronize()
        hp, hl = c.policy(pp, 0.75, return_logits=True)
        hv = c.value(pv)
        only = c.policy(pp, 0.75)
    assert np.array_equal(hp, probs.cpu().numpy()) and np.array_equal(only, hp)
    assert np.array_equal(hl, logits.cpu().numpy())
    assert np.array_equal(hv, value.cpu().numpy())
