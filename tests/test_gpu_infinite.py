"""Infinite and zero operands in the FP64 kernels whose quotients share a
denominator's reciprocal: an infinite time step and infinite updates through
the column hooks, infinite states through the equation of state and the panel
ghosts.  The oracle divides; results are its own bit for bit, NaN where it has
NaN."""
import numpy as np
import pytest

from _columns import column_problem
from exocubed_b200 import CubedSphereAtmosphere
from exocubed_b200 import _native as nat
from exocubed_b200 import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = 3


def _same(got, want):
    bad = ~((got == want) | (np.isnan(got) & np.isnan(want)))
    assert not bad.any(), (int(bad.sum()), got[bad][:4], want[bad][:4])


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("dt,at", [(np.inf, None), (60., 0), (60., 1), (60., 4), (np.inf, 1),
                                   (60., "rho"), (60., "v1"), (60., "v2"), (60., "p")])
def test_column_hooks(oracle_mod, native, full, dt, at):
    ncol, L = 37, 9
    w, du, colgeo, x1f, x1v, dx1f, cfg = column_problem(oracle_mod, ncol, L, seed=3)
    if isinstance(at, str):  # some columns' primitives
        w[5:7, ["rho", "v1", "v2", "", "p"].index(at), G + 4] = np.inf, -np.inf
    elif at is not None:  # some columns' updates; the others stay finite
        du[5, at, 4] = np.inf
        du[33, at, 0] = -np.inf
        du[36, at, L - 1] = np.inf
    want = oracle_mod.implicit_columns(w, du, colgeo, x1f, x1v, dx1f, dt, cfg["gamma"],
                                       cfg["grav"], full=full)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
         for a in (w, du, colgeo, x1f, x1v, dx1f)]
    scratch = torch.empty(ncol * L * 30, dtype=torch.float64, device="cuda")
    hook = native.lib().exo_implicit_columns if full else \
        native.lib().exo_partial_correction_columns
    assert hook(ncol, L, *[a.data_ptr() for a in t], dt, cfg["gamma"], cfg["grav"],
                scratch.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert np.isfinite(want[:5]).all()
    _same(t[1].cpu().numpy(), want)


def _config(setup):
    if setup == "shallow":
        return W.shallow_water_config(N=8, L=3), W.shallow_water_state
    return W.dry_atmosphere_config(N=8, L=6), W.dry_atmosphere_state


def _infinite(setup):
    return [(n, x) for n in ((0, 2, 3) if setup == "shallow" else (0, 2, 3, 4))
            for x in (np.inf, -np.inf)]


@pytest.mark.parametrize("setup", ["shallow", "dry"])
def test_equation_of_state(oracle_mod, setup):
    cfg, make = _config(setup)
    o = oracle_mod.Oracle(cfg)
    o.set_primitive(make(cfg, seed=1))
    u = o.conserved()
    for at, (n, x) in enumerate(_infinite(setup)):
        u[:, n, G + at % 8, G + at // 8, G] = x
    ranges = (G, G + cfg["L"] - 1, G, G + 7, G, G + 7)
    want, _ = o.eos(True, u, ranges)
    with CubedSphereAtmosphere(cfg) as a:
        ud = torch.from_numpy(u).cuda()
        out = torch.zeros_like(ud)
        nat.check(nat.lib().exo_conserved_to_primitive(a._ctx, ud.data_ptr(), out.data_ptr(),
                                                       *ranges, None))
        a.synchronize()
        _same(out.cpu().numpy(), want)


@pytest.mark.parametrize("setup", ["shallow", "dry"])
def test_panel_ghosts(oracle_mod, setup):
    cfg, make = _config(setup)
    for n, x in _infinite(setup):
        w = make(cfg, seed=2)
        W.interior(w)[2, n, 1, 3, 1] = x
        o = oracle_mod.Oracle(cfg)
        o.set_primitive(w)
        with CubedSphereAtmosphere(cfg) as a:
            a.set_primitive(w)
            _same(W.interior(a.conserved()), W.interior(o.conserved()))
            _same(a.primitive(), o.primitive())
