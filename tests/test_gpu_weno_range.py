"""WENO5 of large values: the FP64 build's divisions without range checks hold
for values and differences below 2^200; past that it divides as the oracle
does, bit for bit (values whose differences are small or zero among them)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_large_values_bitwise(oracle_mod, native):
    rng = np.random.default_rng(11)
    rows = [np.full(5, s * x) for x in (1e59, 1.7e60, 1e100, 1e293, 1e294, 1e295, 1e300, 9e307,
                                        1.7e308) for s in (1., -1.)]
    for x in (1e55, 2. ** 199.9, 2. ** 200, 2. ** 201, 1e100, 1e200, 1e294, 1e300, 1.7e308):
        for eps in (0., 1e-15, 1e-9, 1e-3):
            rows += [x * (1. - eps * rng.random(5)) for _ in range(8)]
    x = np.array(rows).T
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in x]
    out = torch.zeros(x.shape[1], dtype=torch.float64, device="cuda")
    assert native.lib().exo_weno5(x.shape[1], *[t.data_ptr() for t in d], out.data_ptr(),
                                  None) == 0
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        want = np.array([oracle_mod.interp_weno5(*c) for c in x.T])
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
