"""Small batches of 128-wide 16-bit nets (a cluster of CTAs a board) against
the same positions in a batch of 256 (the persistent trunk): the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 7, 19, 35, 36, 37, 40)


def _device(c, pp, pv, lo, n):
    import torch
    s = torch.cuda.current_stream().cuda_stream
    p, l = torch.empty((n, 361), device="cuda"), torch.empty((n, 361), device="cuda")
    v = torch.empty(n, device="cuda")
    c.policy_device(pp[lo:].data_ptr(), n, p.data_ptr(), 0.8, l.data_ptr(), s)
    c.value_device(pv[lo:].data_ptr(), n, v.data_ptr(), s)
    torch.cuda.synchronize()
    assert c.device_error() == 0
    return [t.cpu().numpy() for t in (p, l, v)]


@pytest.mark.parametrize("prec", ["bf16", "fp16", "fp8w"])
@pytest.mark.parametrize("n3x3", [1, 2, 11])
def test_clusters_give_the_trunk_bits(gpu_lib, oracle_mod, positions, prec, n3x3):
    """Few and many layers (either row buffer last), every board of a launch,
    sizes on both sides of what fits side by side, one after another."""
    import torch
    lg, O = gpu_lib, oracle_mod
    net = dict(c_in=24, width1=128, width=128, n3x3=n3x3, head_k=1, act=O.RELU, act_head=0)
    pol = O.he_weights(O.make_net(dict(net, value_head=0, fc_hidden=0, value_map=0)), 3)
    val = O.he_weights(O.make_net(dict(net, value_head=1, fc_hidden=64, value_map=0)), 4)
    pp = torch.from_numpy(np.ascontiguousarray(positions["planes_p"][:256, :24])).cuda()
    pv = torch.from_numpy(np.ascontiguousarray(positions["planes_v"][:256, :24])).cuda()
    args = (24, 128, 128, n3x3, 1, lg.LG_ACT_RELU, 0)
    with lg.Context(policy=lg.NetDesc(pol, *args, 0, precision=prec),
                    value=lg.NetDesc(val, *args, 1, 64, 0, precision=prec), max_batch=256) as c:
        for B in SIZES + (256,):
            c.set_tuning(B, 3, 0)
        whole = _device(c, pp, pv, 0, 256)
        for n in SIZES:
            lo = (37 * n) % 200
            for a, b in zip(whole, _device(c, pp, pv, lo, n)):
                assert np.array_equal(a[lo:lo + n], b), n


@pytest.mark.parametrize("act", ["RELU", "ELU"])
def test_chunks_of_clusters(gpu_lib, oracle_mod, positions, act):
    """A device call over chunks that each run in clusters (packing and finish
    as programmatic dependents around them), a ragged last one; ELU nets keep
    the trunk."""
    import torch
    lg, O = gpu_lib, oracle_mod
    net = dict(c_in=24, width1=128, width=128, n3x3=2, head_k=1, act=getattr(O, act), act_head=0)
    pol = O.he_weights(O.make_net(dict(net, value_head=0, fc_hidden=0, value_map=0)), 3)
    val = O.he_weights(O.make_net(dict(net, value_head=1, fc_hidden=64, value_map=0)), 4)
    pp = torch.from_numpy(np.ascontiguousarray(positions["planes_p"][:200, :24])).cuda()
    pv = torch.from_numpy(np.ascontiguousarray(positions["planes_v"][:200, :24])).cuda()
    args = (24, 128, 128, 2, 1, lg.LG_ACT_ELU if act == "ELU" else lg.LG_ACT_RELU, 0)
    kw = dict(policy=lg.NetDesc(pol, *args, 0, precision="bf16"),
              value=lg.NetDesc(val, *args, 1, 64, 0, precision="bf16"))
    with lg.Context(max_batch=200, **kw) as c:
        whole = _device(c, pp, pv, 0, 200)
    with lg.Context(max_batch=30, **kw) as c:
        for n in (200, 67, 30, 4):
            for a, b in zip(whole, _device(c, pp, pv, 0, n)):
                assert np.array_equal(a[:n], b), n
