"""The student kernel with one board a CTA (an SM for every board) and with
pairs of boards gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3x3", [1, 5])
def test_single_boards_and_pairs_give_the_same_bits(gpu_lib, positions, n3x3):
    import torch
    from leela_gb300 import distill
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = 2 * sms + 3
    st = distill.Student(n3x3=n3x3, max_batch=1)
    st.init_he(2)
    params = st.get_params()
    st.close()
    planes = torch.from_numpy(np.ascontiguousarray(positions["planes_p"][:B, :24])).cuda()
    with distill.FastNet(params, n3x3=n3x3, max_batch=B) as f:
        def run(n):
            p, l = torch.empty((n, 361), device="cuda"), torch.empty((n, 361), device="cuda")
            v, e = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
            f.device(planes.data_ptr(), n, p.data_ptr(), v.data_ptr(), 0.8, l.data_ptr(), e.data_ptr())
            f.status()
            return [t.cpu().numpy() for t in (p, l, v, e)]

        whole = run(B)
        for n in (1, 2, sms, sms + 1, 2 * sms + 1):
            for a, b in zip(whole, run(n)):
                assert np.array_equal(a[:n], b), n
