"""The integer-pipe functions on the device (their seeds are the hardware's,
unlike the host build's) against the correctly rounded ones."""
import numpy as np
import pytest

from quijibo_gb300 import lib

pytestmark = pytest.mark.gpu
RANGES = {"exp": (-30.0, 30.0), "log": (1e-6, 1e6), "sin": (0.01, 40.0), "cos": (0.01, 40.0),
          "acos": (2.0 ** -16 - 1, 1 - 2.0 ** -16), "sqrt": (1e-8, 1e4), "rcp": (1e-4, 1e4)}


@pytest.mark.parametrize("name", sorted(RANGES))
def test_device_functions_round_correctly_but_for_a_few(name):
    import torch
    lo, hi = RANGES[name]
    x = torch.rand(200_000, dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    x = (lo * (hi / lo) ** x if lo > 1e-9 and name in ("log", "sqrt", "rcp") else lo + (hi - lo) * x).cuda()
    y, z = torch.empty_like(x), torch.empty_like(x)
    lib.crmath_eval("fx_" + name, x.data_ptr(), y.data_ptr(), x.numel())
    if name in lib.CRM_FUNCTIONS:
        lib.crmath_eval(name, x.data_ptr(), z.data_ptr(), x.numel())
    else:
        z = x.sqrt() if name == "sqrt" else 1.0 / x
    torch.cuda.synchronize()
    y, z = y.cpu().numpy(), z.cpu().numpy()
    big = np.abs(z) > 2.0 ** -4 if name in ("log", "sin", "cos") else np.ones(len(z), bool)
    # 0.53 ulp: at most one unit in the last place, on a few arguments
    assert np.all(np.abs(y - z)[big] <= np.spacing(np.abs(z[big])))
    assert np.mean(y[big] != z[big]) < 0.04
    assert np.all(np.abs(y - z)[~big] <= 2.0 ** -56)
