"""A kernel's error status is reported once, with the call or batch whose
kernels gave up, also while torch's default stream is busy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _busy():
    """Some tens of milliseconds of work on torch's default stream."""
    import torch
    a = torch.randn((8192, 8192), device="cuda", dtype=torch.bfloat16)
    for _ in range(60):
        a = a @ a * 1e-2
    return a


def _context(lg, weights, max_batch):
    return lg.Context(policy=lg.NetDesc.config1_policy(weights["cfg_p"][1], "bf16"),
                      value=lg.NetDesc.config1_value(weights["cfg_v"][1], "bf16"), max_batch=max_batch)


# results by one kernel, and by copies
@pytest.mark.parametrize("B", [4, 40])
def test_the_call_after_a_failed_one_is_good(gpu_lib, weights, positions, B):
    import torch
    lg = gpu_lib
    x = positions["planes_p"][:B, :24]
    with _context(lg, weights, 64) as c:
        c.set_tuning(B, 3, 0)
        good = c.policy(x)
        _busy()
        torch.cuda.synchronize()
        c.inject_stall(0, 1 << 10)
        keep = _busy()
        with pytest.raises(lg.LeelaGPUError) as e:
            c.policy(x)
        assert e.value.code == -5  # LG_ERR_DEVICE
        assert np.array_equal(c.policy(x), good)
        torch.cuda.synchronize()
        assert c.device_error() == 0
        del keep


def test_the_batch_after_a_failed_one_is_good(gpu_lib, weights, positions):
    """The server's first batch gets the error of a device call before it (the
    same context's), the batch behind it its results."""
    import torch
    lg = gpu_lib
    pp, pv = (np.ascontiguousarray(positions[k][:16, :24]) for k in ("planes_p", "planes_v"))
    with _context(lg, weights, 64) as c:
        c.set_tuning(16, 3, 0)
        good = c.value(pv)
        planes, probs = torch.from_numpy(pp).cuda(), torch.empty((16, 361), device="cuda")
        outs = [np.zeros((16, 361), np.float32), np.zeros(16, np.float32)]

        def both():
            c.submit(lg.LG_NET_POLICY, pp, outs[0], tag=1)
            c.submit(lg.LG_NET_VALUE, pv, outs[1], tag=2)
            tags = []
            for _ in range(200):
                tags += c.poll(4, timeout_us=10000)
                if len(tags) == 2:
                    break
            assert sorted(tags) == [1, 2]

        both()  # the server's graphs are there
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            c.inject_stall(0, 1 << 10)
            c.policy_device(planes.data_ptr(), 16, probs.data_ptr(), 1.0, None, side.cuda_stream)
        side.synchronize()
        keep = _busy()
        outs[1][:] = -7.0
        both()
        with pytest.raises(lg.LeelaGPUError):
            c.poll(4)
        assert np.array_equal(outs[1], good)
        assert c.poll(4) == []
        torch.cuda.synchronize()
        assert c.device_error() == 0
        del keep
