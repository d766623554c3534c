"""The second level of a layer reuses the first one's table values where
pressure and temperature agree: same water, same water bin, another bin, and
levels that differ in everything, mixed within a column, against the oracle."""
import numpy as np
import pytest

import oracle
from helpers import compare, mixed_errors, to_numpy
from mgcm_rt import abi, synth

pytestmark = pytest.mark.gpu


def _columns(L):
    b = synth.make_batch(9, L=L, seed=23, cloud=True, night_frac=0.2)
    rng = np.random.default_rng(5)
    lev = 2 * L + 3
    for c in range(9):
        for l in range(1, L + 1):
            k = 2 * l            # index of K = 2l+1; K = 2l+2 follows
            kind = rng.integers(0, 5)
            if kind == 1:        # same bin, another value
                b["qh2o"][c, k:k + 2] = 3.0e-4, 7.0e-4
            elif kind == 2:      # another bin
                b["qh2o"][c, k:k + 2] = 3.0e-4, 3.0e-3
            elif kind == 3:      # off both ends of the water grid
                b["qh2o"][c, k:k + 2] = 0.0, 0.5
            elif kind == 4:      # every coordinate differs
                b["pmid"][c, k + 1] *= 1.3
                b["tmid"][c, k + 1] += 4.0
    assert b["qh2o"].shape[1] == lev
    return b


@pytest.mark.parametrize("L", [1, 2, 24, 48])
def test_layer_gathers_match_oracle(data_dir, otables, L):
    b = _columns(L)
    ref = oracle.run_batch(otables, b)
    rt = abi.Radiation(data_dir, max_layers=L, precision=abi.FP64)
    err = compare(b, to_numpy(rt.run(b)), ref, 1e-12)
    rt.close()
    assert max(err.values()) <= 1e-12, err
    rt = abi.Radiation(data_dir, max_layers=L, precision=abi.MIXED)
    e = mixed_errors(b, rt.run(b), ref)
    rt.close()
    assert e["flux_max"] <= 1e-3 and e["heat_dT_Ksol_max"] <= 1e-2, e
