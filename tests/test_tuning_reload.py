"""A reloaded tuning table runs the kernels that the context which tuned runs,
at every batch size, and tables of other kernels are not taken."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 8, 9, 16, 20, 24)


def _results(c, positions):
    out = []
    for B in SIZES:
        out.append(c.policy(positions["planes_p"][:B], 1.0, return_logits=True)[1])
        out.append(c.value(positions["planes_v"][:B]))
    return out


def test_reload_of_an_fp32_table(gpu_lib, weights, positions, tmp_path):
    """max_batch 24 is no power of two: sizes 17 to 24 are in no bucket that the
    tuner measured, and the file holds none for them."""
    lg = gpu_lib
    path = tmp_path / "tune.json"
    kw = dict(policy=lg.NetDesc.reference_policy(weights["ref_p"][1]),
              value=lg.NetDesc.reference_value(weights["ref_v"][1]), max_batch=24)
    with lg.Context(**kw) as c:
        untuned = _results(c, positions)
        c.autotune(str(path))
        tuned = _results(c, positions)
        table = [c.tuning(B) for B in SIZES]
    saved = json.loads(path.read_text())
    assert set(saved["table"]) == {"1", "2", "4", "8", "16"}
    with lg.Context(**kw) as c:
        c.autotune(str(path))
        assert json.loads(path.read_text()) == saved  # loaded, nothing measured
        assert [c.tuning(B) for B in SIZES] == table
        assert all(np.array_equal(a, b) for a, b in zip(_results(c, positions), tuned))
    # sizes 20 and 24 run the default in both
    assert all(np.array_equal(a, b) for a, b in zip(tuned[-4:], untuned[-4:]))


def test_tables_of_earlier_kernels_are_not_loaded(gpu_lib, weights, positions, tmp_path):
    lg = gpu_lib
    path = tmp_path / "tune.json"
    kw = dict(policy=lg.NetDesc.reference_policy(weights["ref_p"][1]),
              value=lg.NetDesc.reference_value(weights["ref_v"][1]), max_batch=4)
    with lg.Context(**kw) as c:
        c.autotune(str(path))
    saved = json.loads(path.read_text())
    text = path.read_text()
    old = text.replace(saved["key"], saved["key"].split("|mb")[0] + "|mb4")
    assert old != text
    path.write_text(old)
    with lg.Context(**kw) as c:
        c.autotune(str(path))
    assert json.loads(path.read_text())["key"] == saved["key"]
