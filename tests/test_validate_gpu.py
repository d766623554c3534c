"""Input checks of the device calls: a bad value anywhere in an input array is
reported, whichever part of the staging reads it.  The values planted turn
into an error status before the radiation uses them as an index: every table
index is clamped."""
import numpy as np
import pytest

from mgcm_rt import abi, synth

pytestmark = pytest.mark.gpu

LEV_ARRAYS = ("plev", "tlev", "pmid", "tmid", "qh2o", "tauref", "qextrefdst", "taurefcld", "qextrefcld")
BAND_ARRAYS = ("qxvdst", "qsvdst", "gvdst", "qxidst", "qsidst", "gidst",
               "qxvcld", "qsvcld", "gvcld", "qxicld", "qsicld", "gicld")
COL_ARRAYS = ("acosz", "als", "albi", "pcol", "detau")


@pytest.mark.parametrize("solver", [abi.SOLVER_AUTO, abi.SOLVER_FUSED])
@pytest.mark.parametrize("L", [1, 24])
def test_every_input_value_is_checked(data_dir, solver, L):
    import torch
    b = synth.make_batch(6, L=L, seed=91, cloud=True, night_frac=0.5)
    rt = abi.Radiation(data_dir, max_layers=L, precision=abi.FP64, solver=solver)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v
           for k, v in b.items()}

    def status(name, index, value):
        x = dict(dev, **{name: dev[name].clone()})
        x["detau"], x["cumtauv"] = x["detau"].clone(), dev["cumtauv"].clone()
        x[name][index] = value
        try:
            rt.run(x)
        except abi.RTError as e:
            return e.code
        return 0

    assert status("als", 0, 0.25) == 0
    for name in LEV_ARRAYS + BAND_ARRAYS + COL_ARRAYS:
        a = b[name]
        ends = {(c,) + tuple(s) for c in (0, a.shape[0] - 1)
                for s in ([0] * (a.ndim - 1), [n - 1 for n in a.shape[1:]])}
        for index in sorted(ends):
            for bad in (np.nan, -np.inf):
                assert status(name, index, bad) == -2, (name, index, bad)
    for name in ("plev", "pmid"):
        for k in (0, L, 2 * L + 2):
            assert status(name, (3, k), 0.0) == -2, (name, k)
    for k in (0, 1, L + 2, 2 * L + 2):
        assert status("tlev", (5, k), 49.0) == -3, k
        assert status("tlev", (5, k), 900.0) == 0, k     # INT(900*10-499) = 8501, the table's last entry
        assert status("tlev", (5, k), 900.1) == -3, k
    rt.close()
