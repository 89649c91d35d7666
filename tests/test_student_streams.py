"""Student calls on its own stream (stream None, or the default stream's 0)
come after what torch's default stream holds, and before what follows there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _busy():
    """Some tens of milliseconds of work on the current stream."""
    import torch
    a = torch.randn((8192, 8192), device="cuda", dtype=torch.bfloat16)
    for _ in range(40):
        a = a @ a * 1e-2
    return a


@pytest.mark.parametrize("stream", [None, 0])
def test_calls_are_ordered_with_the_default_stream(gpu_lib, positions, stream):
    import torch
    from leela_gb300 import distill
    assert torch.cuda.current_stream().cuda_stream == 0
    B = 32
    rng = np.random.default_rng(1)
    t = rng.random((B, 361)).astype(np.float32) ** 4
    t /= t.sum(1, keepdims=True)
    src = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for a in (positions["planes_p"][:B, :24], t, rng.uniform(-0.8, 0.8, B).astype(np.float32))]
    dst = [torch.zeros_like(a) for a in src]
    ptr = lambda ts: [x.data_ptr() for x in ts]
    st = distill.Student(n3x3=2, max_batch=B)
    st.init_he(3)
    start = st.get_params()
    probs, value = torch.zeros((B, 361), device="cuda"), torch.zeros(B, device="cuda")

    def forward(ts):
        st.forward(ts[0].data_ptr(), B, probs.data_ptr(), value.data_ptr(), stream)
        return probs.cpu().numpy(), value.cpu().numpy()

    def step(ts, want_loss):
        p, t, v = ptr(ts)
        return st.train_step(p, B, t, v, 1e-3, 0.5, stream=stream, want_loss=want_loss)

    def late():
        for d in dst:
            d.zero_()
        torch.cuda.synchronize()
        keep = _busy()
        for d, s in zip(dst, src):
            d.copy_(s)
        return keep

    torch.cuda.synchronize()
    good = forward(src)
    (kl, mse), _ = st.grads(*ptr(src)[:1], B, *ptr(src)[1:], 0.5)
    loss = step(src, True)
    torch.cuda.synchronize()
    after = st.get_params()
    st.set_params(start)

    keep = late()
    probs.zero_()
    value.zero_()
    assert all(np.array_equal(a, b) for a, b in zip(forward(dst), good))
    keep = late()
    (kl2, mse2), _ = st.grads(*ptr(dst)[:1], B, *ptr(dst)[1:], 0.5)
    # (a batch's losses are added up in no fixed order)
    assert np.allclose((kl2, mse2), (kl, mse), rtol=1e-5)
    keep = late()
    assert np.allclose(step(dst, True), loss, rtol=1e-5)
    # the parameters are read after the step that is still running
    st.set_params(start)
    keep = late()
    step(dst, False)
    moved = st.get_params()
    assert np.mean(np.abs(moved - after) > 1e-5) < 1e-2 and not np.array_equal(moved, start)
    del keep
    st.close()


def test_train_steps_see_their_own_minibatches(gpu_lib, positions):
    """train() on torch's default stream gives what the same steps give with a
    synchronization between them."""
    import torch
    from leela_gb300 import distill
    N, batch, steps = 256, 64, 6
    rng = np.random.default_rng(1)
    t = rng.random((N, 361)).astype(np.float32) ** 4
    t /= t.sum(1, keepdims=True)
    planes, t, v = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
                    for a in (positions["planes_p"][:N, :24], t, rng.uniform(-0.8, 0.8, N).astype(np.float32))]
    got = []
    for whole in (True, False):
        st = distill.Student(n3x3=2, max_batch=batch)
        st.init_he(3)
        if whole:
            log = distill.train(st, planes, t, v, steps, batch, seed=5, log_every=1000)
        else:
            g = torch.Generator(device="cpu").manual_seed(5)
            for _ in range(steps):
                idx = torch.randint(0, N, (batch,), generator=g).cuda()
                b = [a.index_select(0, idx).contiguous() for a in (planes, t, v)]
                torch.cuda.synchronize()
                loss = st.train_step(b[0].data_ptr(), batch, b[1].data_ptr(), b[2].data_ptr(), 1e-3, 1.0, want_loss=True)
        got.append(st.get_params())
        st.close()
    assert np.allclose(log[-1][1:], loss, rtol=1e-3)
    assert np.mean(np.abs(got[0] - got[1]) > 1e-4) < 2e-2
