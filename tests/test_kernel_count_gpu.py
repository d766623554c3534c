"""The kernels a call launches, as stats() counts them."""
import pytest

from mgcm_rt import abi
from test_budget_gpu import _tracers, tables  # noqa: F401

pytestmark = pytest.mark.gpu


def _kernels(tables, b, **kw):
    rt = abi.Radiation(tables, max_layers=24, precision=abi.FP64, **kw)
    try:
        rt.run_tracers(b, inplace=True)
        return rt.stats()["kernels"]
    finally:
        rt.close()


def _cloudy(n):
    import torch
    b = _tracers(n, 24)
    clear = torch.zeros((n, 24), dtype=torch.float64, device="cuda")
    return dict(b, cloudon=1, ice_mass=clear, ice_core_mass=clear.clone(), ice_number=clear.clone())


@pytest.mark.parametrize("n", [4000, 16200])
def test_fused_tracer_calls_run_unsplit(tables, n):
    """As many kernels as for a few columns."""
    few = _kernels(tables, _cloudy(60), solver=abi.SOLVER_FUSED)
    assert _kernels(tables, _cloudy(n), solver=abi.SOLVER_FUSED) == few


def test_aerosol_kernel_counted_where_it_runs(tables):
    """Prescribed dust and clear skies have no aerosol optics to compute."""
    assert _kernels(tables, _cloudy(60)) == _kernels(tables, _tracers(60, 24)) + 1
