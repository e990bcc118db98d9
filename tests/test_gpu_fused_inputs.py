"""The mixed 5x5 solve's two ways to load its inputs (level tiles at 64 columns
a block, per lane elsewhere), at the edges of the rule between them: 74 and 85
blocks, 99 and 100 levels, a last warp with 24 columns, and levels that fill no
tile of four.  Every tile gives the same bits, and the oracle's solve."""
import numpy as np
import pytest

from exocubed_b200 import CubedSphereAtmosphere
from exocubed_b200 import _native as nat
from exocubed_b200 import workloads as W

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# FP64 blocks in another order of operations than the oracle's: rounding (2e-16)
# times the blocks' condition (dt |J| of some tens, squared by the elimination)
# stays below 1e-11 of the update.
@pytest.mark.parametrize("N,L", [(28, 33), (30, 1), (30, 6), (30, 33), (30, 99), (30, 100)])
def test_both_ways_give_the_same_solve(oracle_mod, N, L):
    cfg = W.dry_atmosphere_config(N=N, L=L, rsolver=2, implicit_flag=9)
    o = oracle_mod.Oracle(cfg)
    state = W.dry_atmosphere_state(cfg, seed=N + L)
    o.set_primitive(state)
    w = o.primitive()
    rng = np.random.default_rng(N + L)
    scale = np.abs(W.interior(w)).mean(axis=(0, 2, 3, 4))
    du = np.zeros_like(w)
    W.interior(du)[...] = 1e-4 * scale[None, :, None, None, None] * \
        rng.standard_normal(W.interior(du).shape)
    W.interior(du)[:, 1:4] = 1e-3 * rng.standard_normal(W.interior(du)[:, 1:4].shape)
    want = du.copy()
    o.solve_implicit_3d(want, w, 60.0)
    want = W.interior(want)
    got = []
    with CubedSphereAtmosphere(dict(cfg, precision=nat.EXO_PREC_MIXED)) as a:
        a.set_primitive(state)
        for tile in (64, 32, 128):
            a.set_tiles([0, 0, 0, tile, 0, 0])
            x = du.copy()
            a.solve_implicit_3d(x, w, 60.0)
            got.append(W.interior(x).copy())
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    for n in range(5):
        rel = np.linalg.norm(got[0][:, n] - want[:, n]) / np.linalg.norm(want[:, n])
        assert rel < 1e-11, (n, rel)
