"""Contexts and students that just fitted before the tensor-core FP32 kernels
had buffers of their own still do: the buffers shrink or stay out."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _leaving(n):
    """All of the device's free memory taken but n bytes."""
    import torch
    hog = torch.empty((_free() - n) // (2 * MIB) * 2 * MIB, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


# short by less than half of the split trunk's buffers (374 MB at 512 positions
# of width 128), and by nearly all of them
@pytest.mark.parametrize("short", [120, 330])
def test_context_with_little_memory(gpu_lib, oracle_mod, positions, short):
    lg, O = gpu_lib, oracle_mod
    shape = dict(c_in=24, width1=128, width=128, n3x3=2, head_k=1, act=O.RELU, act_head=0, value_head=0, fc_hidden=0,
                 value_map=0)
    w = O.he_weights(O.make_net(shape), 3)
    desc = lambda: lg.NetDesc(w, 24, 128, 128, 2, 1, lg.LG_ACT_RELU, 0, 0)
    x = positions["planes_p"][:300, :24]
    with lg.Context(policy=desc(), max_batch=512) as c:
        c.policy(x)
    before = _free()  # (what the library keeps once loaded is there now)
    with lg.Context(policy=desc(), max_batch=512) as c:
        need = before - _free()
        _, good = c.policy(x, 1.0, return_logits=True)
    with _leaving(need - short * MIB), lg.Context(policy=desc(), max_batch=512) as c:
        _, got = c.policy(x, 1.0, return_logits=True)
    assert np.array_equal(got, good)


def test_student_with_little_memory(gpu_lib, positions):
    import torch
    from leela_gb300 import distill
    B = 512
    rng = np.random.default_rng(1)
    t = rng.random((B, 361)).astype(np.float32) ** 4
    t /= t.sum(1, keepdims=True)
    p, t, v = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
               for a in (positions["planes_p"][:B, :24], t, rng.uniform(-0.8, 0.8, B).astype(np.float32))]

    def grads():
        st = distill.Student(n3x3=2, max_batch=B)
        try:
            st.init_he(3)
            need = before - _free()
            return need, st.grads(p.data_ptr(), B, t.data_ptr(), v.data_ptr(), 0.5)[1]
        finally:
            st.close()

    before = _free()
    grads()
    before = _free()
    need, good = grads()
    with _leaving(need - 150 * MIB):  # of 200 for the backward's buffers
        _, got = grads()
    assert np.linalg.norm(got - good) <= 1e-5 * np.linalg.norm(good)


def test_a_failed_creation_leaves_no_error_behind(gpu_lib, weights, positions):
    import torch
    from leela_gb300 import distill
    lg = gpu_lib
    x = positions["planes_p"][:8]
    kw = dict(policy=lg.NetDesc.reference_policy(weights["ref_p"][1]))
    with lg.Context(max_batch=8, **kw) as c:
        good = c.policy(x)
    for make in (lambda: lg.Context(max_batch=4096, **kw), lambda: distill.Student(max_batch=2048)):
        with _leaving(512 * MIB):
            with pytest.raises(lg.LeelaGPUError) as e:
                make()
        assert e.value.code == -2, str(e.value)  # LG_ERR_ALLOC
        with lg.Context(max_batch=8, **kw) as c:
            planes, probs = torch.from_numpy(x).cuda(), torch.empty((8, 361), device="cuda")
            c.policy_device(planes.data_ptr(), 8, probs.data_ptr(), 1.0)
            torch.cuda.synchronize()
            assert np.array_equal(probs.cpu().numpy(), good)
