"""Parity of the CUDA path (through the C ABI) with the CPU oracle.

Tolerances:
  * shallow water (exo2): bit-exact.  Every device operation there is an IEEE
    +, -, *, / or sqrt evaluated in the oracle's order without fused
    multiply-add, and every transcendental comes from the same host tables.
  * ideal gas (exo3): the hydrostatic decomposition calls log, exp and pow,
    whose CUDA and glibc implementations may differ in the last bit, so
    fluxes and states are compared with a relative tolerance (1e-11 on one
    flux evaluation, 1e-9 relative L2 after a few steps); everything that
    does not depend on the decomposition is still bit-exact.
"""
import ctypes

import numpy as np
import pytest

from exocubed_b200 import workloads as W
from exocubed_b200.atmosphere import CubedSphereAtmosphere

pytestmark = pytest.mark.gpu
G = 3


def _noncorner(a):
    """Cells whose (k,j) is interior or in a ghost band (corners excluded)."""
    nc3, nc2 = a.shape[2], a.shape[3]
    k = np.arange(nc3)[:, None]
    j = np.arange(nc2)[None, :]
    kin = (k >= G) & (k < nc3 - G)
    jin = (j >= G) & (j < nc2 - G)
    m = kin | jin
    return a[:, :, m, :]


def _pair(oracle_mod, cfg, state):
    o = oracle_mod.Oracle(cfg)
    o.set_primitive(state)
    g = CubedSphereAtmosphere(cfg)
    g.set_primitive(state)
    return o, g


def _faces(a, d, L, N):
    """Faces computed on both sides: i interior, face index ranges per dir."""
    if d == 0:
        return a[:, :, G:G + N, G:G + N, G:G + L + 1]
    if d == 1:
        return a[:, :, G:G + N, G:G + N + 1, G:G + L]
    return a[:, :, G:G + N + 1, G:G + N, G:G + L]


@pytest.mark.parametrize("N", [8, 12])
def test_shallow_water_initial_state_bitwise(oracle_mod, N):
    cfg = W.shallow_water_config(N=N)
    state = W.shallow_water_state(cfg, seed=3)
    o, g = _pair(oracle_mod, cfg, state)
    assert np.array_equal(W.interior(g.conserved()), W.interior(o.conserved()))
    assert np.array_equal(_noncorner(g.primitive()), _noncorner(o.primitive()))
    assert g.dt == o.dt


def test_shallow_water_fluxes_bitwise(oracle_mod):
    N = 12
    cfg = W.shallow_water_config(N=N)
    o, g = _pair(oracle_mod, cfg, W.shallow_water_state(cfg, seed=4))
    o.calculate_fluxes()
    g.calculate_fluxes()
    for d in (1, 2):
        a = _faces(g.flux(d), d, 3, N)
        b = _faces(o.flux(d), d, 3, N)
        assert np.array_equal(a, b), f"dir {d}: max diff {np.abs(a - b).max()}"


@pytest.mark.parametrize("rsolver", [0, 3])
def test_shallow_water_steps_bitwise(oracle_mod, rsolver):
    N = 12
    cfg = W.shallow_water_config(N=N, rsolver=rsolver)
    o, g = _pair(oracle_mod, cfg, W.shallow_water_state(cfg, seed=5))
    o.step(3)
    g.step(3)
    assert g.dt == o.dt
    assert g.time == o.time
    ug, uo = W.interior(g.conserved()), W.interior(o.conserved())
    assert np.array_equal(ug[:, [0, 2, 3]], uo[:, [0, 2, 3]]), np.abs(ug - uo).max()
    assert np.array_equal(_noncorner(g.primitive()), _noncorner(o.primitive()))


def test_shallow_water_fixed_dt_many_steps_bitwise(oracle_mod):
    N = 8
    cfg = W.shallow_water_config(N=N)
    o, g = _pair(oracle_mod, cfg, W.shallow_water_state(cfg, seed=6))
    o.step(10, 300.0)
    g.step(10, 300.0)
    assert g.time == o.time == 3000.0
    assert np.array_equal(W.interior(g.conserved())[:, [0, 2, 3]],
                          W.interior(o.conserved())[:, [0, 2, 3]])


@pytest.mark.parametrize("seed", [0, 1])
def test_c1_config_100_steps_bitwise(oracle_mod, seed):
    """The exo2 configuration as specified: 6 x 48 x 48, Roe, CFL 0.4,
    100 steps on the CFL time step, bit-compared with the oracle (conserved
    state, primitives incl. ghosts, time step and time)."""
    cfg = W.shallow_water_config(N=48)
    o, g = _pair(oracle_mod, cfg, W.shallow_water_state(cfg, seed=seed))
    o.step(100)
    g.step(100)
    assert g.dt == o.dt and g.time == o.time
    ug, uo = W.interior(g.conserved()), W.interior(o.conserved())
    assert np.isfinite(ug).all()
    assert np.array_equal(ug[:, [0, 2, 3]], uo[:, [0, 2, 3]]), np.abs(ug - uo).max()
    assert np.array_equal(_noncorner(g.primitive()), _noncorner(o.primitive()))


@pytest.mark.parametrize("L", [12, 32])   # lines that straddle groups of 32, and that fill them
@pytest.mark.parametrize("rsolver", [1, 2])
def test_dry_atmosphere_fluxes(oracle_mod, rsolver, L):
    N = 8
    cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=rsolver)
    o, g = _pair(oracle_mod, cfg, W.dry_atmosphere_state(cfg, seed=7))
    assert np.array_equal(_noncorner(g.primitive()), _noncorner(o.primitive()))
    o.calculate_fluxes()
    g.calculate_fluxes()
    # horizontal fluxes do not touch log/exp/pow: bit-exact
    for d in (1, 2):
        assert np.array_equal(_faces(g.flux(d), d, L, N), _faces(o.flux(d), d, L, N))
    a, b = _faces(g.flux(0), 0, L, N), _faces(o.flux(0), 0, L, N)
    scale = np.abs(b).max(axis=(0, 2, 3, 4), keepdims=True)
    assert np.abs(a - b).max() <= 1e-11 * scale.max()
    assert (np.abs(a - b) / scale).max() < 1e-11


@pytest.mark.parametrize("rsolver", [1, 2])
def test_dry_atmosphere_steps(oracle_mod, rsolver):
    N, L = 8, 12
    cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=rsolver)
    o, g = _pair(oracle_mod, cfg, W.dry_atmosphere_state(cfg, seed=8))
    o.step(3)
    g.step(3)
    ug, uo = W.interior(g.conserved()), W.interior(o.conserved())
    for n in range(5):
        rel = np.linalg.norm(ug[:, n] - uo[:, n]) / np.linalg.norm(uo[:, n])
        assert rel < 1e-9, (n, rel)
    assert g.dt == pytest.approx(o.dt, rel=1e-9)
    assert g.invalid() == 0


def test_implicit_solver_without_decomposition_bitwise(oracle_mod):
    # zero gravity removes log/exp/pow from the step: the 5x5 block solve,
    # Roe averages and eigenvectors are bit-exact
    N, L = 8, 10
    cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=2, grav=0.0)
    o, g = _pair(oracle_mod, cfg, W.dry_atmosphere_state(cfg, seed=9))
    o.step(2, 50.0)
    g.step(2, 50.0)
    assert np.array_equal(W.interior(g.conserved()), W.interior(o.conserved()))


def test_invalid_state_flag(oracle_mod):
    cfg = W.dry_atmosphere_config(N=8, L=8)
    state = W.dry_atmosphere_state(cfg, seed=1)
    state[2, 4, G + 3, G + 3, G + 2] = -5.0   # negative pressure in the input
    g = CubedSphereAtmosphere(cfg)
    g.set_primitive(state)
    assert g.invalid() == 1
    assert g.invalid() == 0  # sticky flag cleared by the read


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("rs,eqn", [(0, 0), (3, 0), (1, 1), (2, 1)])
@pytest.mark.parametrize("ivx", [1, 2, 3])
def test_riemann_rows_bitwise(oracle_mod, native, rs, eqn, ivx):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(10 + rs * 3 + ivx)
    n = 257
    nv = 4 if eqn == 0 else 5
    wl = np.zeros((nv, n))
    wr = np.zeros((nv, n))
    if eqn == 0:
        wl[0] = 2.9e4 * (1 + 0.05 * rng.standard_normal(n))
        wr[0] = 2.9e4 * (1 + 0.05 * rng.standard_normal(n))
    else:
        wl[0] = 1.0 + 0.1 * rng.random(n)
        wr[0] = 1.0 + 0.1 * rng.random(n)
        wl[4] = 1e5 * (1 + 0.1 * rng.random(n))
        wr[4] = 1e5 * (1 + 0.1 * rng.random(n))
        wl[1] = 20 * rng.standard_normal(n)
        wr[1] = 20 * rng.standard_normal(n)
    for q in (2, 3):
        wl[q] = 30 * rng.standard_normal(n)
        wr[q] = 30 * rng.standard_normal(n)
    cosf = 0.4 * rng.standard_normal(n).clip(-1.5, 1.5) / 1.5
    sinf = np.sqrt(1 - cosf ** 2)
    cthp = cosf * (1 + 1e-12)
    cthc = 0.3 * rng.standard_normal(n).clip(-2, 2) / 2
    d = [_dev(torch, x) for x in (wl, wr, np.zeros((nv, n)), cosf, sinf, cthp, cthc)]
    rc = native.lib().exo_riemann(rs, eqn, ivx, n, 1.4, *[t.data_ptr() for t in d], None)
    assert rc == 0
    torch.cuda.synchronize()
    got = d[2].cpu().numpy()
    for m in range(n):
        a = np.zeros(5)
        b = np.zeros(5)
        a[:nv] = wl[:, m]
        b[:nv] = wr[:, m]
        ref = oracle_mod.riemann_face(rs, eqn, ivx, 1.4, a, b, cosf[m], sinf[m], cthp[m], cthc[m])
        assert np.array_equal(got[:, m], ref[:nv]), (m, got[:, m], ref[:nv])


def test_weno5_rows_bitwise(oracle_mod, native):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    n = 1000
    args = [rng.standard_normal(n) * 10 ** rng.uniform(-3, 3, n) for _ in range(5)]
    d = [_dev(torch, a) for a in args] + [_dev(torch, np.zeros(n))]
    assert native.lib().exo_weno5(n, *[t.data_ptr() for t in d], None) == 0
    torch.cuda.synchronize()
    got = d[5].cpu().numpy()
    ref = np.array([oracle_mod.interp_weno5(*(a[m] for a in args)) for m in range(n)])
    assert np.array_equal(got, ref)
    one = [_dev(torch, np.array([float(x)])) for x in (1, 2, 3, 4, 5)] + [_dev(torch, np.zeros(1))]
    native.lib().exo_weno5(1, *[t.data_ptr() for t in one], None)
    torch.cuda.synchronize()
    assert one[5].cpu().numpy()[0] == 2.5000000000000004
