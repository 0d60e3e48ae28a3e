"""Where a small channel's Poisson solve takes one launch and where the three passes:
the launches of a step on both sides of each line of the rule, with its measured
reason, and the same bits either way."""
import numpy as np
import pytest

from test_gpu_row_forms import start

pytestmark = pytest.mark.gpu

F64, F32 = 0, 1
# nx, ny, storage, launches a step: 2 (LBM, solve) or 4 (LBM, three passes); in
# brackets the time of a step with one launch over that with three, on B200
RULE = [
    (10, 101, F64, 2),    # 0.89
    (2, 400, F64, 2),     # 0.89: 200 row pairs, 13 a block, one round
    (2, 700, F64, 4),     # 1.08: two rounds
    (2, 4000, F64, 4),    # 1.58
    (27, 400, F32, 2),    # FP32 storage, FP64 solve
    (27, 570, F32, 4),
    (10, 256, F64, 2),    # 0.91: column segments of 4 rows
    (10, 300, F64, 4),    # 1.07: of 5
    (50, 130, F64, 2),    # 0.88: of 4
    (50, 131, F64, 4),    # of 5
    (50, 259, F64, 2),    # 0.91: of 9
    (64, 128, F32, 2),    # 0.99
    (16, 258, F32, 2),    # 0.93: segments of 4 rows
    (16, 259, F32, 4),    # 1.08: of 5
    (256, 20, F32, 4),    # 1.07
    (16, 128, F64, 2),    # 0.84
    (32, 128, F64, 4),    # 1.04
    (64, 128, F64, 4),    # 1.07
    (1000, 12, F64, 2),   # 0.98
    (1500, 6, F64, 4),    # 1.02
    (131, 34, F64, 2),    # 0.81: one row pair a block of a prime length
    (131, 35, F64, 4),    # 1.05 at 48 rows
]


@pytest.mark.parametrize("nx,ny,storage,per_step", RULE)
def test_launches_of_a_step(nx, ny, storage, per_step):
    import ekpnp
    p, init = start(nx, ny, storage)
    out = []
    for profile in (False, True):
        with ekpnp.Channel(p) as ch:
            ch.set_fields(**init)
            ch.init_equilibrium()
            ch.step(1)
            ch.profile(profile)
            before = ch.launches
            ch.step(10)
            if not profile:
                # FP32 storage with the FP64 solve: its right-hand side and its psi are converted
                extra = 2 if storage == F32 and (nx & (nx - 1) or nx < 16) else 0
                assert ch.launches - before == 10 * (per_step + extra)
            out.append(ch.get_fields())
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
