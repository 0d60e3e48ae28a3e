"""The row transforms and the step at lengths where their forms can go wrong:
mixed-radix lengths (every butterfly, prime radices, primes, tiny lengths),
two-nodes-a-thread steps of odd and very narrow channels, and the step's
launch chain against one step a call."""
import numpy as np
import pytest

from conftest import rel_err
from test_oracle import _numpy_poisson

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [2, 3, 4, 5, 6, 7, 9, 12, 25, 49, 60, 97, 105, 143, 243, 625, 1000, 1009, 1331, 2047])
@pytest.mark.parametrize("ny", [4, 9])
def test_mixed_radix_poisson_matches_numpy(nx, ny):
    import ekpnp
    p = ekpnp.channel_params(nx, ny, kappa_h=5.0, zeta=-1.5, zeta_hi=-0.7)
    rng = np.random.default_rng(nx * 7 + ny)
    cp = 1.0 + 0.1 * rng.standard_normal((ny, nx))
    cn = 1.0 + 0.1 * rng.standard_normal((ny, nx))
    with ekpnp.Channel(p) as ch:
        ch.set_fields(cp=cp, cn=cn)
        ch.poisson()
        got = ch.get_fields(("psi", "ex", "ey"))
    phi, ex, ey = _numpy_poisson(p, cp, cn, p["zeta_lo"], p["zeta_hi"])
    # the bar of test_gpu_poisson_matches_numpy
    assert rel_err(got["psi"], phi) < 1e-12
    assert np.abs(got["ex"] - ex).max() < 1e-12 * np.abs(phi).max()
    assert np.abs(got["ey"] - ey).max() < 1e-12 * np.abs(phi).max()


def start(nx, ny, storage, seed=3, **kw):
    import ekpnp
    p = ekpnp.channel_params(nx, ny, kappa_h=4.0, zeta=-1.0, ex=5e-4, eps=0.1, storage=storage, **kw)
    return p, ekpnp.noisy_uniform_state(nx, ny, seed)


def run(p, init, calls):
    import ekpnp
    with ekpnp.Channel(p) as ch:
        ch.set_fields(**init)
        ch.init_equilibrium()
        for n in calls:
            ch.step(n)
        return ch.get_fields()


@pytest.mark.parametrize("nx,ny", [(2, 9), (3, 12), (5, 33), (15, 20), (16, 7), (17, 5), (31, 40), (33, 21), (255, 11), (257, 9)])
def test_fp32_step_of_odd_and_narrow_channels(nx, ny):
    """FP32 against FP64 within 1e-5 of max-abs, every row (the bar of the
    shifted-storage tests), after 60 steps of a channel with asymmetric walls
    and a moving top wall."""
    kw = dict(zeta_hi=-0.6, uw=1e-3)
    init = start(nx, ny, 0)[1]
    a = run(start(nx, ny, 0, **kw)[0], init, [60])
    b = run(start(nx, ny, 1, **kw)[0], init, [60])
    for k in ("rho", "ux", "cp", "cn", "psi"):
        assert np.abs(a[k] - b[k]).max() <= 1e-5 * np.abs(a[k]).max(), k


# 512 x 513 lies above the node count up to which the step's kernels are chained
@pytest.mark.parametrize("nx,ny", [(10, 101), (64, 20), (512, 513)])
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32", "f16"])
def test_chained_steps_equal_single_steps(nx, ny, storage):
    """One call of n steps (kernels launched as a chain) gives the bits of n
    calls of one step (each starting with an ordinary launch)."""
    p, init = start(nx, ny, storage)
    a, b = run(p, init, [24]), run(p, init, [1] * 24)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("nx,ny", [(16, 4), (16, 401), (32, 33), (64, 128), (128, 17), (256, 31), (2, 9), (10, 101), (97, 12),
                                   (100, 150), (128, 65), (512, 12)])
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32", "f16"])
def test_one_launch_solve_equals_the_passes(nx, ny, storage):
    """A small channel's Poisson solve in one launch gives the bits of the
    three passes (which profiling runs by themselves), at both sides of the
    node count up to which it is taken."""
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


# at and around 2^20 nodes, with partial last blocks (odd widths, one column over) and the last rows
@pytest.mark.parametrize("nx,ny", [(1024, 1023), (1024, 1024), (1025, 1033), (131, 8100), (8192, 130)])
def test_prefetching_step_equals_the_pipelined_one(nx, ny):
    """The large FP16 step that prefetches later blocks' rows gives the bits of
    the TMA-fed kernel."""
    import ekpnp
    p, init = start(nx, ny, 2)
    out = []
    for form in ("plain", "tma"):
        with ekpnp.Channel(p) as ch:
            ch.set_lbm_kernel(form)
            ch.set_fields(**init)
            ch.init_equilibrium()
            ch.step(6)
            out.append(ch.get_fields())
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
