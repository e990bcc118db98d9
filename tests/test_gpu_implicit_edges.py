"""The implicit solve at the sizes where its pipeline can go wrong: columns
around the ring's and the level tile's lengths (1 to 9 levels and the next
ones), groups of one column, of 31, 32 and 33.  FP64 against the
oracle bit for bit; the mixed builds against the oracle's FP64 solve."""
import numpy as np
import pytest

from _columns import column_problem
from exocubed_b200 import CubedSphereAtmosphere
from exocubed_b200 import _native as nat
from exocubed_b200 import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("ncol,L", [(1, 1), (31, 2), (32, 3), (33, 4), (64, 5), (65, 6), (3, 7),
                                    (40, 8), (97, 9), (5, 12), (32, 13), (2, 250)])
def test_column_hooks_bitwise(oracle_mod, native, full, ncol, L):
    w, du, colgeo, x1f, x1v, dx1f, cfg = column_problem(oracle_mod, ncol, L, seed=L + ncol)
    want = oracle_mod.implicit_columns(w, du, colgeo, x1f, x1v, dx1f, 60., cfg["gamma"],
                                       cfg["grav"], full=full)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
         for a in (w, du, colgeo, x1f, x1v, dx1f)]
    # canaries: the hook may use ncol*L*30 doubles of scratch and no more
    scratch = torch.full((ncol * L * 30 + 64,), 7., dtype=torch.float64, device="cuda")
    hook = native.lib().exo_implicit_columns if full else \
        native.lib().exo_partial_correction_columns
    rc = hook(ncol, L, *[a.data_ptr() for a in t], 60., cfg["gamma"], cfg["grav"],
              scratch.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0, native.lib().exo_last_error()
    assert np.array_equal(t[1].cpu().numpy(), want)
    assert bool((scratch[ncol * L * 30:] == 7.).all())


# FP64 blocks take the same blocks in another order of operations: rounding
# (2e-16) times the blocks' condition (dt |J| of some tens, squared by the
# elimination) stays below 1e-11 of the update.  FP32 blocks: 6e-8 times the
# same, 1e-3 with a margin of three for the deepest column.
@pytest.mark.parametrize("precision,tol", [(nat.EXO_PREC_MIXED, 1e-11),
                                           (nat.EXO_PREC_MIXED_F32_SOLVE, 1e-3)])
@pytest.mark.parametrize("implicit", [9, 1])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 8, 9, 21, 64])
def test_mixed_solve_matches_the_oracle(oracle_mod, precision, tol, implicit, L):
    cfg = W.dry_atmosphere_config(N=6, L=L, rsolver=2, implicit_flag=implicit)
    o = oracle_mod.Oracle(cfg)
    state = W.dry_atmosphere_state(cfg, seed=L)
    o.set_primitive(state)
    w = o.primitive()
    rng = np.random.default_rng(L)
    scale = np.abs(W.interior(w)).mean(axis=(0, 2, 3, 4))
    du = np.zeros_like(w)
    W.interior(du)[...] = 1e-4 * scale[None, :, None, None, None] * \
        rng.standard_normal(W.interior(du).shape)
    W.interior(du)[:, 1:4] = 1e-3 * rng.standard_normal(W.interior(du)[:, 1:4].shape)
    want, got = du.copy(), du.copy()
    o.solve_implicit_3d(want, w, 60.0)
    with CubedSphereAtmosphere(dict(cfg, precision=precision)) as a:
        a.set_primitive(state)
        a.solve_implicit_3d(got, w, 60.0)
    want, got = W.interior(want), W.interior(got)
    for n in range(5):
        rel = np.linalg.norm(got[:, n] - want[:, n]) / np.linalg.norm(want[:, n])
        assert rel < tol, (n, rel)
    if implicit == 1:
        assert np.array_equal(got[:, 2:4], W.interior(du)[:, 2:4])
