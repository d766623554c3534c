"""Systems whose operands leave the range of the solves' fast arithmetic take
the general solve: same results as the oracle (1e-12, the FP64 tolerance),
alone and beside ordinary columns of the same warp."""
import numpy as np
import pytest

import oracle
from helpers import compare, to_numpy
from mgcm_rt import abi, synth

pytestmark = pytest.mark.gpu


def _ordinary(b, c):
    pass


def _unit_asymmetry_ir(b, c):      # COSBI = 1
    b["gidst"][c] = 1.0


def _wide_asymmetry_vis(b, c):     # COSBV > 1 where dust outweighs Rayleigh scattering
    b["gvdst"][c, :, 20:40] = 1.01


def _subnormal_dust(b, c):         # a scattering numerator below 2^-300
    b["tauref"][c] *= 1e-305


def _opaque_dust(b, c):            # DTAU above 2^100
    b["tauref"][c, 30:40] = 1e40


def _huge_cosine(b, c):            # cos(zenith) above 2^30
    b["acosz"][c] = 1e12


def _no_scattering_vis(b, c):      # W0 near 0 (Rayleigh only)
    b["qsvdst"][c] = 0.0


@pytest.mark.parametrize("L", [1, 24, 36])
@pytest.mark.parametrize("plant", [_ordinary, _unit_asymmetry_ir, _wide_asymmetry_vis, _subnormal_dust,
                                   _opaque_dust, _huge_cosine, _no_scattering_vis])
def test_out_of_range_systems_match_oracle(data_dir, otables, plant, L):
    b = synth.make_batch(5, L=L, seed=17, cloud=False, night_frac=0.0)
    for c in (1, 4):
        plant(b, c)
    ref = oracle.run_batch(otables, b)
    assert all(np.isfinite(v).all() for v in ref.values())
    rt = abi.Radiation(data_dir, max_layers=L, precision=abi.FP64)
    err = compare(b, to_numpy(rt.run(b)), ref, 1e-12)
    rt.close()
    assert max(err.values()) <= 1e-12, err
