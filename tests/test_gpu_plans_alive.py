"""Channels of several lengths alive at once.  All mixed-radix lengths share
their row kernels, and the small ones the one-launch solve: what one channel's
creation, or a solve without allocation, sets on a kernel must leave the
others' launches allowed."""
import numpy as np
import pytest

from test_gpu_row_forms import start
from test_zz_no_alloc import charges, noalloc_solve

pytestmark = pytest.mark.gpu


def channel(nx, ny, storage):
    import ekpnp
    p, init = start(nx, ny, storage)
    ch = ekpnp.Channel(p)
    ch.set_fields(**init)
    ch.init_equilibrium()
    return ch


def alone(nx, ny, storage, calls):
    with channel(nx, ny, storage) as ch:
        for n in calls:
            ch.step(n)
        return ch.get_fields()


def same(got, want):
    for k in want:
        assert np.array_equal(got[k], want[k]), k


# the row passes (above 16384 nodes), and the solve in one launch (below): 1000 x
# 16 and 100 x 150 ask for 64,000 and 51,200 bytes of shared memory there, 300 x 50
# for 38,400, 10 x 101 for 5,120
@pytest.mark.parametrize("a,b", [((2047, 12), (10, 1700)), ((1000, 257), (6, 3000)), ((1000, 16), (10, 101)),
                                 ((100, 150), (10, 101)), ((300, 50), (10, 101)), ((2047, 12), (10, 101))])
@pytest.mark.parametrize("storage", [0, 1], ids=["f64", "f32"])
def test_two_lengths_alive(a, b, storage):
    """Steps of two channels in turn, the longer rows' channel created first
    and last, give the bits of each channel by itself."""
    calls = [3, 2]
    want = {s: alone(*s, storage, calls) for s in (a, b)}
    for order in ((a, b), (b, a)):
        chans = {s: channel(*s, storage) for s in order}
        for n in calls:
            for s in order:
                chans[s].step(n)
        for s in order:
            same(chans[s].get_fields(), want[s])
            chans[s].close()


@pytest.mark.parametrize("nx,ny", [(2047, 12), (1000, 16), (1000, 257)])
def test_noalloc_solve_between_steps(nx, ny):
    """A solve without allocation of a short length between the steps of a
    channel of long rows, and one of that length after them."""
    import ekpnp
    calls = [3, 2]
    want = alone(nx, ny, 0, calls)
    small = ekpnp.channel_params(10, 20, kappa_h=3.0, zeta=-1.0)
    big = ekpnp.channel_params(nx, ny, kappa_h=3.0, zeta=-1.0)
    first = noalloc_solve(big, *charges(nx, ny, 5, 0.2))
    with channel(nx, ny, 0) as ch:
        for n in calls:
            noalloc_solve(small, *charges(10, 20, 6, 0.1))
            ch.step(n)
        same(ch.get_fields(), want)
    noalloc_solve(small, *charges(10, 20, 6, 0.1))
    same(noalloc_solve(big, *charges(nx, ny, 5, 0.2)), first)
