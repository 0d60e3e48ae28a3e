"""FP64 divisions by a channel's constants at the edges of the range: constants
whose reciprocal overflows or is subnormal, and an electric field of psi with
infinite, overflowing and subnormal differences."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# accepted by ek_create (eps: any but zero); 1 / 1e-310 overflows, 1 / 1e308 is subnormal
@pytest.mark.parametrize("name,value", [("eps", 1e-310), ("eps", -1e-310), ("eps", 1e308), ("dx", 1e-310), ("dx", 1e308)])
@pytest.mark.parametrize("nx,ny", [(10, 21), (32, 17)])
def test_steps_with_extreme_constants_match_the_oracle(oracle_mod, name, value, nx, ny):
    """Uncharged ions between grounded walls: psi and E are exactly zero, and so is
    every dividend of the extreme constant; the flow and the diffusion go on."""
    import ekpnp
    p = ekpnp.channel_params(nx, ny, kappa_h=4.0, zeta=0.0, uw=1e-3)
    p.update({name: value, "f_charge": 0.0})
    init = ekpnp.noisy_uniform_state(nx, ny, 5)
    init["psi"] = np.zeros((ny, nx))
    steps = 20
    with ekpnp.Channel(p) as ch:
        ch.set_fields(**init)
        ch.init_equilibrium()
        ch.step(steps)
        got = ch.get_fields()
    o = oracle_mod.OracleChannel(p)
    o.set_fields(**init)
    o.init_equilibrium()
    o.step(steps)
    want = o.get_fields()
    # densities of 1: the bar of the parity tests.  Velocities are differences of
    # populations below 1: steps x 9 populations x 4 roundings of 2^-53
    for k in ("rho", "ux", "uy", "cp", "cn", "psi", "ex", "ey"):
        assert np.all(np.isfinite(want[k])), k
        bar = steps * 9 * 4 * 2.0 ** -53 if k in ("ux", "uy") else 1e-12 * np.abs(want[k]).max()
        assert np.abs(got[k] - want[k]).max() <= bar, k


@pytest.mark.parametrize("dx,dy", [(3.0, 7.0), (0.1, 1e-3), (1e-310, 1e308)])
@pytest.mark.parametrize("storage", [0, 1], ids=["f64", "f32"])
def test_field_of_extreme_potentials_is_the_division(dx, dy, storage):
    """E = 0.5 (psi - psi') / spacing, bit for bit as numpy divides."""
    import ekpnp
    nx, ny = 12, 9
    rng = np.random.default_rng(1)
    psi = rng.standard_normal((ny, nx)) * 10.0 ** rng.integers(-323, 308, (ny, nx))
    psi[1, 1], psi[2, 5], psi[4, 4:7], psi[6, :3] = np.inf, -np.inf, 1.7e308, 5e-324
    psi[7, 2:9] = 0.25
    p = dict(ekpnp.channel_params(nx, ny, kappa_h=4.0, zeta=-1.0, storage=storage), dx=dx, dy=dy)
    with ekpnp.Channel(p) as ch:
        ch.set_fields(psi=psi)
        got = ch.get_fields(("ex", "ey"))
    yc = np.clip(np.arange(ny), 1, ny - 2)
    with np.errstate(all="ignore"):
        ex = 0.5 * (np.roll(psi, 1, 1) - np.roll(psi, -1, 1)) / dx
        ey = 0.5 * (psi[yc - 1] - psi[yc + 1]) / dy
    for k, e in (("ex", ex), ("ey", ey)):
        nan = np.isnan(e)
        assert np.array_equal(np.isnan(got[k]), nan), k
        assert np.array_equal(got[k][~nan].view(np.int64), e[~nan].view(np.int64)), k
