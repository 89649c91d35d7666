"""The student's gradients on the tensor cores against the FP64 oracle at the
sizes where tiles, row ranges and channel blocks end; and the wide FFMA tiles
of its forward against the narrow ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,c_in,n3x3", [
    (1, 24, 1),    # seven row stages, fewer row ranges than CTAs
    (2, 25, 2),    # 125 of the first layer's 128 expanded channels
    (17, 7, 3),    # a ragged last stage (6,800 L3 rows)
    (33, 24, 5),   # the served shape
    (3, 26, 1),    # 130 expanded channels: the FFMA kernels
])
def test_gradients_vs_fp64(gpu_lib, B, c_in, n3x3):
    import torch
    from leela_gb300 import distill
    from oracle import distill_oracle as D
    rng = np.random.default_rng(B)
    st = distill.Student(c_in=c_in, n3x3=n3x3, max_batch=B)
    st.init_he(4)
    planes = (rng.random((B, c_in, 361)) < 0.2).astype(np.uint8)
    t = rng.random((B, 361)).astype(np.float32) ** 4
    t /= t.sum(1, keepdims=True)
    vt = rng.uniform(-0.8, 0.8, B).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (planes, t, vt)]
    _, g = st.grads(dev[0].data_ptr(), B, dev[1].data_ptr(), dev[2].data_ptr(), 0.5)
    _, g64 = D.loss_and_grads(st.get_params(), planes, t, vt, 0.5, c_in, 64, n3x3, 64)
    floor = 1e-4 * np.abs(g64).max()
    off = 0
    for s in D.shapes(c_in, 64, n3x3, 64):
        sizes = [s[3] * s[2] * s[1] * s[1], s[3]] if s[0] == "conv" else [s[1]]
        for n in sizes:
            a, b = g[off:off + n], g64[off:off + n]
            off += n
            # (2e-3: an activation within rounding of zero may fall on either side)
            assert np.abs(a - b).max() / max(np.abs(b).max(), floor) <= 2e-3, (s, n)
    st.close()


@pytest.mark.parametrize("width,sizes", [(64, (53, 54, 109, 163, 217)), (192, (17, 18, 37, 55, 73))])
def test_wide_ffma_tiles_give_the_same_bits(gpu_lib, oracle_mod, width, sizes):
    """The 16 x 8-output FFMA kernel over ragged batches whose shares end in one
    to four 64-row blocks: the same bits at each size, and at the size just
    under its first (64 x 64 tiles, K split) the same but for the order of
    FP32 sums."""
    lg, O = gpu_lib, oracle_mod
    shape = dict(c_in=24, width1=width, width=width, n3x3=2, head_k=1, act=O.RELU, act_head=0, value_head=0,
                 fc_hidden=0, value_map=0)
    w = O.he_weights(O.make_net(shape), 6)
    x = (np.random.default_rng(2).random((sizes[-1], 24, 361)) < 0.2).astype(np.uint8)
    with lg.Context(policy=lg.NetDesc(w, 24, width, width, 2, 1, lg.LG_ACT_RELU, 0, 0), max_batch=sizes[-1]) as c:
        for B in sizes:
            c.set_tuning(B, 0, 0)
        _, a = c.policy(x, 1.0, return_logits=True)
        for B in sizes[:-1]:
            _, b = c.policy(x[:B], 1.0, return_logits=True)
            if B == sizes[0]:
                assert np.abs(b - a[:B]).max() <= 1e-5 * np.abs(a).max()
            else:
                assert np.array_equal(a[:B], b), B
