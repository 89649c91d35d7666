"""The FP32 path's error against 64 bits over whole nets, where the split trunk
took the place of the FFMA kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nets", ["cfg", "ref"])
@pytest.mark.parametrize("B", [3, 5, 8, 77])
def test_default_fp32_error(gpu_lib, oracle_mod, weights, positions, nets, B):
    """Logits of the untuned context, relative 2-norm: 7.2e-7 to 7.8e-7 as a mean
    over 24 seeds, 1.04e-6 at most; held to twice that largest one.  The small-
    batch kernel gives 8.9e-7 to 9.3e-7, 1.6e-6 at most."""
    lg, O = gpu_lib, oracle_mod
    n, w = weights[nets + "_p"]
    c_in = 24 if nets == "cfg" else 32
    x = positions["planes_p"][:B, :c_in]
    O.enable_blas()
    try:
        ref = O.forward_f64(n, w, x)
    finally:
        O.disable_blas()
    desc = (lg.NetDesc.config1_policy if nets == "cfg" else lg.NetDesc.reference_policy)(w)
    with lg.Context(policy=desc, max_batch=77) as c:
        _, got = c.policy(x, 1.0, return_logits=True)
    err = _rel(got, ref)
    print(f"{nets} {B}: {err:.2e}")
    assert err <= 2.1e-6
