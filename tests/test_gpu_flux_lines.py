"""The fluxes at the sizes where their lines, chunks and segments can go
wrong (x2/x3: lines that fill no group of 32, faces one past a chunk, one and several
chunks per segment, four variables, both ways of the mixed reconstruction; x1: columns
per block), and WENO5 where its divisions leave the unchecked path."""
import numpy as np
import pytest

from exocubed_b200 import CubedSphereAtmosphere
from exocubed_b200 import _native as nat
from exocubed_b200 import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = 3


def _faces(a, d, N, L):
    k, j = (N, N + 1) if d == 1 else (N + 1, N)
    return a[:, :, G:G + k, G:G + j, G:G + L]


# FP64: every operation of these fluxes is the oracle's, bit for bit.  Mixed
# (its FP32 fluxes are not handed out): density and pressure after a short step
# (a CFL step empties an atmosphere of few levels).  One rounding of the
# pressure (6e-8) moves the face velocity by 6e-8 c / gamma; ten of them over a step of Courant number 0.02 are 1e-8 of the density, while
# a wrong cell's velocity of some m/s against c = 300 m/s is 5e-5.
@pytest.mark.parametrize("setup,N,L", [
    ("dry", 6, 1), ("dry", 6, 9), ("dry", 6, 16), ("dry", 14, 33), ("dry", 16, 45),
    ("dry", 30, 31), ("dry", 32, 40), ("dry", 16, 100), ("dry", 30, 96), ("dry", 6, 250),
    ("shallow", 6, 5), ("shallow", 8, 32), ("shallow", 16, 3), ("shallow", 30, 70)])
def test_horizontal_fluxes_match_the_oracle(oracle_mod, setup, N, L):
    if setup == "dry":
        cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=nat.EXO_RS_HLLC)
        state = W.dry_atmosphere_state(cfg, seed=N + L)
    else:
        cfg = W.shallow_water_config(N=N, L=L)
        state = W.shallow_water_state(cfg, seed=N + L)
    o = oracle_mod.Oracle(cfg)
    o.set_primitive(state)
    o.calculate_fluxes()
    with CubedSphereAtmosphere(cfg) as g:
        g.set_primitive(state)
        g.calculate_fluxes()
        for d in (1, 2):
            got, want = _faces(g.flux(d), d, N, L), _faces(o.flux(d), d, N, L)
            assert np.array_equal(got, want), (d, np.abs(got - want).max())
    o.set_primitive(state)
    if L < G:  # the reflected ghosts of a step need G levels
        return
    dt = 0.05 * o.dt
    o.step(1, dt)
    with CubedSphereAtmosphere(dict(cfg, precision=nat.EXO_PREC_MIXED)) as g:
        g.set_primitive(state)
        g.step(1, dt)
        got, want = W.interior(g.primitive()), W.interior(o.primitive())
    for n in (0, 4) if setup == "dry" else (0,):
        err = np.abs(got[:, n] / want[:, n] - 1.).max()
        assert err < 1e-6, (n, err)


# The decomposition's log, exp and pow are the device's: 1e-11 of the largest
# flux, as for any FP64 x1 flux (columns that fill their block, that leave a
# warp idle, and blocks of more places than threads).
@pytest.mark.parametrize("rsolver", [nat.EXO_RS_LMARS, nat.EXO_RS_HLLC])
@pytest.mark.parametrize("L,columns", [(3, 4), (25, 8), (25, 1), (57, 4), (250, 4), (250, 5),
                                       (121, 8)])
def test_vertical_fluxes_match_the_oracle(oracle_mod, rsolver, L, columns):
    N = 6
    cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=rsolver)
    o = oracle_mod.Oracle(cfg)
    o.set_primitive(W.dry_atmosphere_state(cfg, seed=L))
    o.calculate_fluxes()
    want = o.flux(0)[:, :, G:G + N, G:G + N, G:G + L + 1]
    with CubedSphereAtmosphere(cfg) as g:
        g.set_tiles([columns, 0, 0, 0, 0, 0])
        g.set_primitive(W.dry_atmosphere_state(cfg, seed=L))
        g.calculate_fluxes()
        got = g.flux(0)[:, :, G:G + N, G:G + N, G:G + L + 1]
    scale = np.abs(want).max(axis=(0, 2, 3, 4), keepdims=True)
    assert (np.abs(got - want) / scale).max() < 1e-11


def test_weno5_outside_the_unchecked_divisions_bitwise(oracle_mod, native):
    rng = np.random.default_rng(5)
    rows = [rng.standard_normal(5) * 10. ** e
            for e in (-320, -300, -160, -80, -9, 0, 29, 29.5, 30, 30.25, 30.5, 31, 40, 60, 75, 80,
                      150, 200, 300) for _ in range(20)]
    for bad in (np.nan, np.inf, -np.inf, 1e308, 5e-324, 1e31):
        for at in range(5):
            row = rng.standard_normal(5)
            row[at] = bad
            rows.append(row)
    rows += [np.full(5, x) for x in (0., -0., 1e31, 1e200, np.inf, np.nan)]
    x = np.array(rows).T
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in x]
    out = torch.zeros(x.shape[1], dtype=torch.float64, device="cuda")
    assert native.lib().exo_weno5(x.shape[1], *[t.data_ptr() for t in d], out.data_ptr(),
                                  None) == 0
    torch.cuda.synchronize()
    want = np.array([oracle_mod.interp_weno5(*c) for c in x.T])
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
