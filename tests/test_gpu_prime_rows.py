"""Channels whose length has a prime factor above 5, summed term by term: the kernel
of prime lengths, its launches and its share of the one-launch solve."""
import time

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_row_forms import start
from test_oracle import _numpy_poisson

pytestmark = pytest.mark.gpu


# primes below, at and above a block's threads (256) and its whole warps; the two
# sides of 128 columns and 74 row pairs (ordinary launches); two primes' product and
# a prime with small radices, which stay in the mixed kernel
@pytest.mark.parametrize("nx,ny", [(7, 600), (31, 400), (127, 149), (127, 152), (131, 149), (131, 150), (131, 153), (251, 60),
                                   (257, 61), (509, 40), (1021, 20), (217, 60), (398, 50)])
def test_prime_lengths_match_numpy(nx, ny):
    import ekpnp
    p = ekpnp.channel_params(nx, ny, kappa_h=5.0, zeta=-1.5, zeta_hi=-0.7)
    rng = np.random.default_rng(nx * 7 + ny)
    cp = 1.0 + 0.1 * rng.standard_normal((ny, nx))
    cn = 1.0 + 0.1 * rng.standard_normal((ny, nx))
    with ekpnp.Channel(p) as ch:
        ch.set_fields(cp=cp, cn=cn)
        ch.poisson()
        psi = ch.get_fields(("psi",))["psi"]
    # the bar of test_gpu_poisson_matches_numpy
    assert rel_err(psi, _numpy_poisson(p, cp, cn, p["zeta_lo"], p["zeta_hi"])[0]) < 1e-12


# one and two row pairs a block of the one-launch solve, 256 points and more
@pytest.mark.parametrize("nx,ny", [(113, 64), (127, 66), (131, 34), (131, 35), (251, 34), (251, 36), (401, 34), (31, 200)])
@pytest.mark.parametrize("storage", [0, 1], ids=["f64", "f32"])
def test_one_launch_solve_of_prime_lengths_equals_the_passes(nx, ny, storage):
    import ekpnp
    p, init = start(nx, ny, storage)
    out = []
    for profile in (False, True):
        with ekpnp.Channel(p) as ch:
            ch.set_fields(**init)
            ch.init_equilibrium()
            ch.profile(profile)
            ch.step(12)
            out.append(ch.get_fields())
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


def us_a_step(nx, ny):
    import ekpnp
    p, init = start(nx, ny, 0)
    with ekpnp.Channel(p) as ch:
        ch.set_fields(**init)
        ch.init_equilibrium()
        best = float("inf")
        for _ in range(20):
            t = time.perf_counter()
            ch.step(40)
            ch.sync()
            best = min(best, time.perf_counter() - t)
    return best / 40 * 1e6


# against the power of two beside it, on B200: 131 x 400 takes 2.1 times as long, 4.8
# times with too few threads; 251 x 60 2.8 times, 5.6 so and in one launch
@pytest.mark.parametrize("prime,two,most", [((131, 400), (128, 400), 3.4), ((251, 60), (256, 60), 4.2)])
def test_prime_lengths_use_the_gpu(prime, two, most):
    ratios = []
    for _ in range(3):  # the host can be late, never early
        ratios.append(us_a_step(*prime) / us_a_step(*two))
    assert min(ratios) < most, ratios
