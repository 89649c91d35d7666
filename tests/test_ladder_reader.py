"""The ladder planes against the oracle's reader on boards that games hardly
give: scattered stones (strings in atari everywhere, captures and suicides on
the way) and ladders that run across an empty board, with and without a stone
in their way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LADDER = ((0, 0, 1), (0, 1, 0), (1, 0, 0), (-1, 0, 0), (1, 1, 0), (0, -1, 0))  # dy, dx, colour: 1 runs, 0 hunts


def _alive(sq):
    """sq [19][19] without the strings that have no liberty."""
    seen = np.zeros((19, 19), bool)
    out = sq.copy()
    for y, x in np.argwhere(sq != 2):
        if seen[y, x]:
            continue
        todo, string, free = [(y, x)], [], False
        seen[y, x] = True
        while todo:
            a, b = todo.pop()
            string.append((a, b))
            for c, d in ((a - 1, b), (a + 1, b), (a, b - 1), (a, b + 1)):
                if not (0 <= c < 19 and 0 <= d < 19):
                    continue
                if sq[c, d] == 2:
                    free = True
                elif sq[c, d] == sq[y, x] and not seen[c, d]:
                    seen[c, d] = True
                    todo.append((c, d))
        if not free:
            for a, b in string:
                out[a, b] = 2
    return out


def _boards(n, seed):
    rng = np.random.default_rng(seed)
    sq = np.full((n, 19, 19), 2, np.int8)
    for i in range(n):
        if i % 2 == 0:  # scattered stones
            fill = rng.uniform(0.05, 0.75)
            u = rng.random((19, 19))
            sq[i][u < fill] = 1
            sq[i][u < fill / 2] = 0
        else:  # a stone in atari with room to run, few stones elsewhere
            b = sq[i]
            y, x = rng.integers(2, 17, 2)
            for _ in range(rng.integers(0, 12)):
                b[tuple(rng.integers(0, 19, 2))] = rng.integers(0, 2)
            fy, fx, swap = rng.choice([-1, 1]), rng.choice([-1, 1]), rng.integers(0, 2)
            flip = rng.integers(0, 2)
            keep = rng.integers(4, 7)
            for dy, dx, c in LADDER[:keep]:
                dy, dx = (dx, dy) if swap else (dy, dx)
                b[y + fy * dy, x + fx * dx] = c ^ flip
        sq[i] = _alive(sq[i])
    return sq.reshape(n, 361), rng.integers(0, 2, n).astype(np.int8)


@pytest.mark.parametrize("seed", [1, 2])
def test_ladder_planes_on_scattered_stones(gpu_lib, oracle_mod, seed):
    import torch
    n = 400
    sq, tm = _boards(n, seed)
    mv = np.full((n, 4), -1, np.int32)
    d = [torch.from_numpy(a).cuda() for a in (sq, tm, mv)]
    for which, lad in ((0, 25), (1, 27)):
        out = torch.empty((n, 32, 361), dtype=torch.uint8, device="cuda")
        gpu_lib.gather_device(d[0].data_ptr(), d[1].data_ptr(), n, which, 32, out.data_ptr(), None, d[2].data_ptr())
        torch.cuda.synchronize()
        ref = oracle_mod.gather_planes(sq, tm, which, 32, mv)
        assert ref[:, lad].any() and ref[:, lad + 1].any()
        assert np.array_equal(out.cpu().numpy(), ref)
