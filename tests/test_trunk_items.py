"""The persistent trunk's item sizes (64, 128 or 256 rows by batch) give the
same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "fp16", "fp8w"])
@pytest.mark.parametrize("choice", [2, 3])
def test_item_sizes_give_the_same_bits(gpu_lib, weights, positions, prec, choice):
    """Batches on both sides of each change of item size (24 / 25 and 97 / 98
    positions) and the smallest, against the same positions in a batch of
    256; with the first layer inside the launch and before it."""
    lg = gpu_lib
    pp, pv = positions["planes_p"][:256, :24], positions["planes_v"][:256, :24]
    with lg.Context(policy=lg.NetDesc.config1_policy(weights["cfg_p"][1], prec),
                    value=lg.NetDesc.config1_value(weights["cfg_v"][1], prec), max_batch=256) as c:
        for B in (1, 24, 25, 97, 98, 256):
            c.set_tuning(B, choice, 0)
        _, ref = c.policy(pp, 1.0, return_logits=True)
        vref = c.value(pv)
        for B in (1, 3, 24, 25, 97, 98):
            _, logits = c.policy(pp[:B], 1.0, return_logits=True)
            assert np.array_equal(logits, ref[:B]), B
            assert np.array_equal(c.value(pv[:B]), vref[:B]), B
