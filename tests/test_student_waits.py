"""Waits of the student's kernels that run out: whole warps give up together,
the launch ends in bounded time with an error status, and what follows is as
if it had not been."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one board a CTA; pairs of boards, a second group on some CTAs
@pytest.mark.parametrize("n3x3", [1, 5])
@pytest.mark.parametrize("B", [1, 2 * 152 + 3])
def test_serving_wait_runs_out(gpu_lib, positions, n3x3, B):
    import torch
    from leela_gb300 import distill
    lg = gpu_lib
    st = distill.Student(n3x3=n3x3, max_batch=1)
    st.init_he(2)
    params = st.get_params()
    st.close()
    planes = torch.from_numpy(np.ascontiguousarray(positions["planes_p"][:B, :24])).cuda()
    with distill.FastNet(params, n3x3=n3x3, max_batch=B) as f:
        p, v = torch.empty((B, 361), device="cuda"), torch.empty(B, device="cuda")

        def run():
            f.device(planes.data_ptr(), B, p.data_ptr(), v.data_ptr(), 1.0)
            f.status()
            return [t.cpu().numpy() for t in (p, v)]

        good = run()
        f.inject_stall(1 << 14)
        t0 = time.perf_counter()
        with pytest.raises(lg.LeelaGPUError) as e:
            run()
        elapsed = time.perf_counter() - t0
        assert e.value.code == -5, str(e.value)  # LG_ERR_DEVICE
        assert elapsed < 20.0
        assert all(np.array_equal(a, b) for a, b in zip(run(), good))
        print(f"stalled call returned after {elapsed * 1e3:.1f} ms: {e.value}")


def _batch(positions, B, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    t = rng.random((B, 361)).astype(np.float32) ** 4
    t /= t.sum(1, keepdims=True)
    v = rng.uniform(-0.8, 0.8, B).astype(np.float32)
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (positions["planes_p"][:B, :24], t, v)]


# one row range a tap group; every SM busy
@pytest.mark.parametrize("B", [1, 64])
def test_weight_gradient_wait_runs_out(gpu_lib, positions, B):
    from leela_gb300 import distill
    lg = gpu_lib
    st = distill.Student(n3x3=2, max_batch=B)
    st.init_he(3)
    p, t, v = _batch(positions, B)

    def run():
        return st.grads(p.data_ptr(), B, t.data_ptr(), v.data_ptr(), 0.5)[1]

    good = run()
    st.inject_stall(1 << 14)
    t0 = time.perf_counter()
    with pytest.raises(lg.LeelaGPUError) as e:
        run()
    elapsed = time.perf_counter() - t0
    assert e.value.code == -5, str(e.value)  # LG_ERR_DEVICE
    assert elapsed < 20.0
    # sums over rows are added up in no fixed order
    assert np.abs(run() - good).max() <= 1e-5 * np.abs(good).max()
    print(f"stalled call returned after {elapsed * 1e3:.1f} ms: {e.value}")
    st.close()


@pytest.mark.parametrize("seen_by", ["loss", "step", "forward", "grads", "params"])
def test_failed_training_step_leaves_the_parameters(gpu_lib, positions, seen_by):
    """A step whose weight gradient gave up changes nothing, nor does one after
    it, until a call reports the error; training then goes on as if neither
    had been (Adam's step count included)."""
    import torch
    from leela_gb300 import distill
    lg = gpu_lib
    B = 16
    st = distill.Student(n3x3=2, max_batch=B)
    st.init_he(3)
    p, t, v = _batch(positions, B)
    probs, value = torch.empty((B, 361), device="cuda"), torch.empty(B, device="cuda")

    def step(want_loss=False):
        return st.train_step(p.data_ptr(), B, t.data_ptr(), v.data_ptr(), 1e-3, 0.5, want_loss=want_loss)

    start = st.get_params()
    step(True)
    one = st.get_params()
    step(True)
    two = st.get_params()
    st.set_params(start)
    step(True)
    first = st.get_params()
    st.inject_stall(1 << 14)
    report = {"loss": lambda: step(True), "step": step,
              "forward": lambda: st.forward(p.data_ptr(), B, probs.data_ptr(), value.data_ptr()),
              "grads": lambda: st.grads(p.data_ptr(), B, t.data_ptr(), v.data_ptr(), 0.5),
              "params": st.get_params}[seen_by]
    if seen_by != "loss":
        step()
        torch.cuda.synchronize()
    with pytest.raises(lg.LeelaGPUError) as e:
        report()
    assert e.value.code == -5, str(e.value)  # LG_ERR_DEVICE
    assert np.array_equal(st.get_params(), first)
    step(True)
    # one step moves a parameter by about 1e-3; sums are added up in no fixed
    # order, and a gradient near zero may take either sign of it
    near = lambda a, b: np.mean(np.abs(a - b) > 1e-5) < 1e-2
    assert near(first, one) and near(st.get_params(), two) and not near(one, two)
    st.close()
