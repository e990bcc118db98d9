"""The momenta of the mixed build after a short step, at the sizes where the
x1 and x2/x3 kernels' lines, chunks and columns can go wrong, and shallow water
of one and two layers."""
import numpy as np
import pytest

from exocubed_b200 import CubedSphereAtmosphere
from exocubed_b200 import _native as nat
from exocubed_b200 import workloads as W

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# Scaled by density times sound speed.  The tangential momenta change by
# dt/dx times FP32 fluxes near the pressure rho c^2 / gamma: ten roundings of
# 6e-8 at a Courant number of 0.02 are 1e-8; a component from a wrong cell or
# variable changes them by 0.02 (5 m/s / 300 m/s)^2 = 5e-6.  The vertical one
# sees the FP32 reconstruction of perturbations of 0.4 % of the pressure at
# vertical Courant numbers up to 200: 5e-8; a wrong one changes it by 0.05.
TANGENTIAL, VERTICAL = 2e-7, 1e-5


@pytest.mark.parametrize("setup,N,L", [
    ("dry", 6, 9), ("dry", 6, 16), ("dry", 14, 33), ("dry", 16, 45), ("dry", 30, 31),
    ("dry", 32, 40), ("dry", 16, 100), ("dry", 6, 250),
    ("shallow", 6, 5), ("shallow", 8, 32), ("shallow", 16, 3), ("shallow", 30, 1),
    ("shallow", 16, 2)])
def test_momenta_after_a_short_step(oracle_mod, setup, N, L):
    if setup == "dry":
        cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=nat.EXO_RS_HLLC)
        state = W.dry_atmosphere_state(cfg, seed=N + L)
    else:
        cfg = W.shallow_water_config(N=N, L=L)
        state = W.shallow_water_state(cfg, seed=N + L)
    o = oracle_mod.Oracle(cfg)
    o.set_primitive(state)
    dt = 0.05 * o.dt
    w = W.interior(o.primitive())
    scale = w[:, 0] * np.sqrt(1.4 * w[:, 4] / w[:, 0] if setup == "dry" else w[:, 0])
    o.step(1, dt)
    with CubedSphereAtmosphere(dict(cfg, precision=nat.EXO_PREC_MIXED)) as g:
        g.set_primitive(state)
        g.step(1, dt)
        got, want = W.interior(g.conserved()), W.interior(o.conserved())
    for n, tol in ((1, VERTICAL), (2, TANGENTIAL), (3, TANGENTIAL))[0 if setup == "dry" else 1:]:
        err = np.abs((got[:, n] - want[:, n]) / scale).max()
        assert err < tol, (n, err)
