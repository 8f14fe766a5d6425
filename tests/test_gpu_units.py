"""A passive scalar's results do not depend on its unit (needs a B200).

The row kernels pack two real rows into one complex transform, whose rounding is
relative to the larger of the two.  With a scalar of another size than U1's in the
pair its accuracy would follow from its unit: multiplied by a power of two, it
would come out with other digits.  With the pair's members brought to one
magnitude by powers of two every operation on the scalar scales exactly, so the
scalar's digits, and the velocity's, must stay the same to the last bit; no tolerance.
"""
import math

import numpy as np
import pytest

import oracle as O
from diablo_b200 import configs, ics
from diablo_b200.params import Params

pytestmark = pytest.mark.gpu

SHIFT = (9, -4)  # binary orders that TH1 and TH2 are made smaller by


def run(solver, p, gy, st, times):
    ch = solver(p) if gy is None else solver(p, gy)
    ch.set_state(st)
    ch.set_time(0.0, p.delta_t)
    ch.steps(1, times)
    out = {k: ch.get_field(k).copy() for k in ["CU1", "CU2", "CU3"] +
           ["CTH%d" % n for n in range(p.n_th)]}
    ch.close()
    return out


def check(solver, p, gy, st, times):
    a = run(solver, p, gy, st, times)
    small, q = dict(st), p.replace()
    q.th_bc_ymin_c1, q.th_bc_ymax_c1 = list(p.th_bc_ymin_c1), list(p.th_bc_ymax_c1)
    for n in range(p.n_th):
        f = 2.0 ** -SHIFT[n]
        small["CTH%d" % n] = st["CTH%d" % n] * f
        q.th_bc_ymin_c1[n] *= f
        q.th_bc_ymax_c1[n] *= f
    b = run(solver, q, gy, small, times)
    for k in a:
        f = 2.0 ** SHIFT[int(k[3:])] if k.startswith("CTH") else 1.0
        assert np.isfinite(a[k]).all() and np.abs(a[k]).max() > 0
        assert np.array_equal(a[k], b[k] * f), k


@pytest.mark.parametrize("precision,nx,nz,n_th", [
    (1, 16, 32, 2), (1, 64, 16, 1), (1, 96, 16, 2), (1, 128, 32, 1), (1, 192, 16, 2), (1, 256, 16, 2),
    (1, 384, 16, 1), (1, 512, 16, 1), (1, 512, 16, 2), (0, 30, 18, 1), (0, 128, 54, 1), (0, 160, 18, 2),
    (0, 192, 20, 1), (0, 256, 16, 2), (0, 384, 16, 2), (0, 512, 18, 1)])
def test_channel_scalar_units(precision, nx, nz, n_th):
    from diablo_b200.solver import Channel
    p, gy = configs.channel_re180(nx=nx, ny=11, nz=nz)
    p = p.replace(n_th=n_th, precision=precision, variable_dt=0, delta_t=5e-4)
    p.pr = [0.71, 1.3, 1, 1]
    p.ri = [0.0, 0.0, 0, 0]
    p.th_bc_ymin_c1 = [-1.0, 0.5, 0, 0]
    p.th_bc_ymax_c1 = [1.0, -0.5, 0, 0]
    ref = O.Oracle(p, gy)
    u1, u2, u3, th = ics.channel_laminar(p, gy, seed=5)
    ref.create_flow_chan(u1, u2, u3, th)
    st = ref.state()
    for n in range(n_th):  # the scalars: eddies of U3's and U2's shape on a mean profile
        st["CTH%d" % n] = st["CU3" if n == 0 else "CU2"] + 0.0
        st["CTH%d" % n][:, 0, 0] += np.linspace(-1, 1, p.ny + 2)
    check(Channel, p, gy, st, 2)


@pytest.mark.parametrize("precision,n,n_th", [
    (1, (96, 10, 10), 1), (1, (128, 12, 18), 2), (1, (256, 10, 10), 2), (1, (256, 8, 12), 1),
    (1, (64, 8, 1280), 1), (0, (30, 10, 10), 1), (0, (128, 10, 10), 2), (0, (256, 8, 10), 1),
    (0, (60, 10, 18), 2)])
def test_periodic_scalar_units(precision, n, n_th):
    from diablo_b200.solver import Periodic
    nx, ny, nz = n
    p = Params(nx=nx, ny=ny, nz=nz, num_per_dir=3, nu=0.01, lx=2 * math.pi, ly=2 * math.pi,
               lz=2 * math.pi, delta_t=0.005, variable_dt=0, n_th=n_th, precision=precision)
    p.ri = [0.0, 0.0, 0, 0]
    p.pr = [0.7, 1.5, 1, 1]
    ref = O.Oracle(p, None)
    for nm, a in zip(("CU1", "CU2", "CU3"), ics.periodic_spectrum(p, seed=7)):
        ref.set(nm, a)
    for i in range(n_th):
        ref.set("CTH%d" % i, ics.periodic_spectrum(p, seed=17 + i)[0])
    ref.rem_div_per()
    check(Periodic, p, None, ref.state(), 2)


@pytest.mark.parametrize("precision,nx", [(1, 64), (1, 128), (1, 192), (1, 256), (1, 384), (1, 512),
                                          (0, 30), (0, 128), (0, 192), (0, 512)])
@pytest.mark.parametrize("flow", ["channel", "box"])
def test_scalar_of_zeros_takes_no_rounding_from_u1(flow, precision, nx):
    """A passive scalar of zeros beside U1 counts as 2^60 times smaller (FP64: 2^500), so what U1's
    rounding leaves in its row, at most 2^-20 of U1 per transform, comes out below 2^-80, and
    after 6 substeps that each add less than it times CFL number and 2^9 modes below 2^-60."""
    from diablo_b200.solver import Channel, Periodic
    if flow == "box" and precision and nx in (192, 384, 512):
        pytest.skip("no mixed form of the box")
    if flow == "channel":
        p, gy = configs.channel_re550(nx=nx, ny=17, nz=16)
        p = p.replace(precision=precision)
        p.th_bc_ymin_c1[0] = p.th_bc_ymax_c1[0] = 0.0
        u1, u2, u3, th = ics.channel_laminar(p, gy, seed=3)
        ch = Channel(p, gy)
        ch.create_flow(u1, u2, u3, 0 * th)
    else:
        p = Params(nx=nx, ny=8, nz=10, num_per_dir=3, nu=0.01, lx=2 * math.pi, ly=2 * math.pi,
                   lz=2 * math.pi, delta_t=0.002, variable_dt=0, n_th=1, precision=precision)
        p.ri = [0.0, 0, 0, 0]
        ch = Periodic(p)
        for nm, a in zip(("CU1", "CU2", "CU3"), ics.periodic_spectrum(p, seed=7)):
            ch.set_field(nm, a)
        ch.rem_div_per()
    ch.set_time(0.0, p.delta_t)
    ch.steps(1, 2)
    u, th = ch.get_field("CU1"), ch.get_field("CTH0")
    ch.close()
    assert np.isfinite(th).all() and np.abs(u).max() > 0
    assert np.abs(th).max() <= 2.0 ** (-60 if precision else -500) * np.abs(u).max()
