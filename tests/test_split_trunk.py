"""The FP32 trunk on the tensor cores (each value as the sum of three BF16
parts, kernel choice 3 of FP32 nets) against the FP64 oracle and the FFMA
kernels."""
import numpy as np
import pytest

from conftest import rel_logit_err

pytestmark = pytest.mark.gpu

# norm-wise logit error of a short FP32 net: a few times 2^-24 a layer, with
# room for the worst of some hundred positions
TOL = 5e-6


def _planes(B, c_in, seed, high=2):
    return np.random.default_rng(seed).integers(0, high, (B, c_in, 361)).astype(np.uint8)


@pytest.mark.parametrize("B", [1, 3, 8, 9, 33])
@pytest.mark.parametrize("c_in,width1,width,n3x3,head_k,act", [
    (24, 128, 128, 2, 1, "RELU"),   # the benchmark nets' layers
    (32, 96, 128, 2, 3, "ELU"),     # the reference's policy shape, padded first layer, 3x3 head
    (32, 64, 64, 1, 3, "ELU"),      # one 3x3 layer, one channel group
    (18, 32, 160, 2, 1, "RELU"),    # c_in not a multiple of 8, partial groups
    (13, 130, 33, 3, 1, "ELU"),     # odd channel counts
    (64, 256, 256, 1, 1, "RELU"),   # the widest, five input halves
])
def test_split_trunk_vs_fp64(gpu_lib, oracle_mod, B, c_in, width1, width, n3x3, head_k, act):
    """Shapes at the edges of groups, halves and row tiles, as accurate as
    the FFMA kernels."""
    lg, O = gpu_lib, oracle_mod
    a = getattr(O, act)
    shape = dict(c_in=c_in, width1=width1, width=width, n3x3=n3x3, head_k=head_k, act=a, act_head=0,
                 value_head=0, fc_hidden=0, value_map=0)
    n = O.make_net(shape)
    w = O.he_weights(n, 5)
    x = _planes(B, c_in, B, 2 if B != 3 else 256)
    O.enable_blas()
    try:
        ref = O.forward_f64(n, w, x)
    finally:
        O.disable_blas()
    desc = lg.NetDesc(w, c_in, width1, width, n3x3, head_k, lg.LG_ACT_ELU if act == "ELU" else lg.LG_ACT_RELU, 0, 0)
    with lg.Context(policy=desc, max_batch=33) as c:
        c.set_tuning(B, 3, 0)
        _, split = c.policy(x, 1.0, return_logits=True)
        c.set_tuning(B, 0, 0)
        _, ffma = c.policy(x, 1.0, return_logits=True)
    assert rel_logit_err(split, ref).max() <= TOL
    assert rel_logit_err(ffma, split).max() <= 2 * TOL


def test_split_trunk_is_the_same_at_every_batch(gpu_lib, weights, positions):
    """A position's result does not depend on its batch, on the launch it
    falls into (1,024 positions each) or on what ran before in the same
    buffers, with both nets' widths taking turns."""
    import torch
    lg = gpu_lib
    B = 1030
    planes = {k: torch.from_numpy(np.ascontiguousarray(positions[k][np.arange(B) % 1024])).cuda()
              for k in ("planes_p", "planes_v")}
    with lg.Context(policy=lg.NetDesc.reference_policy(weights["ref_p"][1]),
                    value=lg.NetDesc.reference_value(weights["ref_v"][1]), max_batch=B) as c:
        s = torch.cuda.current_stream().cuda_stream

        def run(lo, n):
            p, l, v = torch.empty((n, 361), device="cuda"), torch.empty((n, 361), device="cuda"), torch.empty(n, device="cuda")
            c.policy_device(planes["planes_p"][lo:].data_ptr(), n, p.data_ptr(), 1.0, l.data_ptr(), s)
            c.value_device(planes["planes_v"][lo:].data_ptr(), n, v.data_ptr(), s)
            torch.cuda.synchronize()
            return [t.cpu().numpy() for t in (p, l, v)]

        whole = run(0, B)
        for lo, n in ((0, 9), (1000, 30), (1021, 9), (500, 3)):
            for a, b in zip(whole, run(lo, n)):
                assert np.array_equal(a[lo:lo + n], b), (lo, n)
        assert c.device_error() == 0


def test_infinite_weights_keep_the_ffma_kernels(gpu_lib, oracle_mod):
    """An infinite weight has no parts: such a net keeps the per-layer
    kernels where nobody chose a kernel."""
    lg, O = gpu_lib, oracle_mod
    shape = dict(c_in=24, width1=64, width=64, n3x3=1, head_k=1, act=O.RELU, act_head=0, value_head=0,
                 fc_hidden=0, value_map=0)
    w = O.he_weights(O.make_net(shape), 5).copy()
    w[7] = np.inf
    x = _planes(12, 24, 1)
    with lg.Context(policy=lg.NetDesc(w, 24, 64, 64, 1, 1, lg.LG_ACT_RELU, 0, 0), max_batch=12) as c:
        _, got = c.policy(x, 1.0, return_logits=True)
        c.set_tuning(12, 0, 0)
        _, ref = c.policy(x, 1.0, return_logits=True)
    assert np.array_equal(got, ref, equal_nan=True)
