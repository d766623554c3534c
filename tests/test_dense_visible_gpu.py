"""Calls on both sides of the size up to which one kernel screens and solves
the visible systems (three columns per SM), day and night columns mixed,
against the oracle: the FP64 outputs to 1e-12, MIXED within its tolerance."""
import numpy as np
import pytest

import oracle
from helpers import compare, mixed_errors, to_numpy
from mgcm_rt import abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 24, 99])
@pytest.mark.parametrize("above", [0, 1])
def test_both_sides_of_the_dense_limit(data_dir, otables, L, above):
    import torch
    n = 3 * torch.cuda.get_device_properties(0).multi_processor_count + above
    b = synth.make_batch(n, L=L, seed=61, cloud=True, night_frac=0.4)
    ref = oracle.run_batch(otables, b)
    for precision in (abi.FP64, abi.MIXED):
        rt = abi.Radiation(data_dir, max_layers=L, precision=precision)
        got = rt.run(b)
        systems = rt.stats()["systems"]
        rt.close()
        assert 0 < systems <= 204 * n
        if precision == abi.FP64:
            err = compare(b, to_numpy(got), ref, 1e-12)
            assert max(err.values()) <= 1e-12, err
        else:
            e = mixed_errors(b, got, ref)
            assert e["flux_max"] <= 1e-3 and e["heat_dT_Ksol_max"] <= 1e-2, e
    assert np.isfinite(ref["qrad"]).all()
