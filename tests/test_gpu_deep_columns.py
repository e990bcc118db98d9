"""The column hooks at the deepest columns they take, against the oracle bit for
bit: the last depth with two warps a block, the first with one, the limit."""
import numpy as np
import pytest

from _columns import column_problem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = 3


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("ncol,L", [(2, 4899), (33, 4900), (33, 5518)])
def test_deepest_columns_bitwise(oracle_mod, native, full, ncol, L):
    w, du, colgeo, x1f, x1v, dx1f, cfg = column_problem(oracle_mod, 33, 50, seed=2)
    rep = -(-L // 50)  # the 50-level columns over and over, spheres of one spacing
    w = np.ascontiguousarray(np.concatenate([w[:ncol, :, :G], np.tile(w[:ncol, :, G:-G], rep)[:, :, :L],
                                             w[:ncol, :, -G:]], axis=2))
    du = np.ascontiguousarray(np.tile(du[:ncol], rep)[:, :, :L])
    x1f = x1f[0] + (x1f[1] - x1f[0]) * np.arange(L + 7) / rep
    x1v, dx1f = 0.5 * (x1f[1:] + x1f[:-1]), np.diff(x1f)
    want = oracle_mod.implicit_columns(w, du, colgeo[:ncol].copy(), x1f, x1v, dx1f, 60.,
                                       cfg["gamma"], cfg["grav"], full=full)
    assert np.isfinite(want).all()
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
         for a in (w, du, colgeo[:ncol], x1f, x1v, dx1f)]
    scratch = torch.empty(ncol * L * 30, dtype=torch.float64, device="cuda")
    hook = native.lib().exo_implicit_columns if full else \
        native.lib().exo_partial_correction_columns
    assert hook(ncol, L, *[a.data_ptr() for a in t], 60., cfg["gamma"], cfg["grav"],
                scratch.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert np.array_equal(t[1].cpu().numpy(), want)
