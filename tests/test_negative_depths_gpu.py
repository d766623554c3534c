"""A layer whose two levels have optical depths of opposite signs, and a
negative depth at level 2: finite inputs that pass the checks, with exponents
of the layers' middles far outside the range of the solves' fast exponential.
The results are the oracle's, infinities and NaN included, in every solve that
has a fast form: small FP64 calls (one kernel screens and solves), large FP64
calls and MIXED ones (a screen and a list), planted columns among ordinary day
and night ones."""
import numpy as np
import pytest

import oracle
from helpers import compare
from mgcm_rt import abi, synth
from test_solve_range_gpu import (_huge_cosine, _no_scattering_vis, _opaque_dust, _ordinary, _subnormal_dust,
                                  _unit_asymmetry_ir, _wide_asymmetry_vis)

pytestmark = pytest.mark.gpu

DUST = ("qextrefdst", "qxvdst", "qsvdst", "gvdst", "qxidst", "qsidst", "gidst")


def _two_signs(lower):
    """Layer L // 2 + 1: 3005 in one level and -3000 in the other, of the same dust."""
    def plant(b, c):
        k = 2 * (int(b["L"]) // 2 + 1)          # index of K = 2l + 1
        for n in DUST:
            b[n][c, ..., k + 1] = b[n][c, ..., k]
        b["tauref"][c, k + 1 - lower], b["tauref"][c, k + lower] = 3005.0, -3000.0
    return plant


def _negative_level2(b, c):
    b["tauref"][c, 1] = -3000.0


NEGATIVE = {"negative_above": _two_signs(0), "negative_below": _two_signs(1), "negative_level2": _negative_level2}
FINITE = {f.__name__: f for f in (_ordinary, _unit_asymmetry_ir, _wide_asymmetry_vis, _subnormal_dust, _opaque_dust,
                                  _huge_cosine, _no_scattering_vis)}


def _batch(n, L, plant):
    b = synth.make_batch(n, L=L, seed=29, cloud=False, night_frac=0.3)
    for c in range(1, n, 3):
        plant(b, c)
    return b


def _large():
    import torch
    return 3 * torch.cuda.get_device_properties(0).multi_processor_count + 5


def _run(data_dir, b, precision):
    rt = abi.Radiation(data_dir, max_layers=int(b["L"]), precision=precision)
    try:
        return {k: np.asarray(v) for k, v in rt.run(b).items()}
    finally:
        rt.close()


def _finite(got, ref):
    """Both with zeros for infinities and NaN, which have to be the same."""
    for k, r in ref.items():
        assert np.array_equal(np.isnan(got[k]), np.isnan(r)), k
        inf = np.isinf(r)
        assert np.array_equal(np.isinf(got[k]), inf) and np.array_equal(got[k][inf], r[inf]), k
    return [{k: np.where(np.isfinite(v), v, 0.0) for k, v in x.items()} for x in (got, ref)]


@pytest.mark.parametrize("L", [2, 24])
@pytest.mark.parametrize("plant", sorted(NEGATIVE))
@pytest.mark.parametrize("large", [False, True])
def test_negative_depths_match_oracle(data_dir, otables, large, plant, L):
    b = _batch(_large() if large else 5, L, NEGATIVE[plant])
    ref = oracle.run_batch(otables, b)
    if plant != "negative_below":      # there the exponent's cap at 35 holds
        assert not all(np.isfinite(v).all() for v in ref.values())
    got, ref = _finite(_run(data_dir, b, abi.FP64), ref)
    err = compare(b, got, ref, 1e-12)
    assert max(err.values()) <= 1e-12, err


@pytest.mark.parametrize("plant", sorted(NEGATIVE))
@pytest.mark.parametrize("large", [False, True])
def test_negative_depths_mixed(data_dir, otables, large, plant):
    """MIXED: infinities and NaN where the oracle has them, and no others."""
    b = _batch(_large() if large else 5, 24, NEGATIVE[plant])
    ref, got = oracle.run_batch(otables, b), _run(data_dir, b, abi.MIXED)
    for k, r in ref.items():
        assert np.array_equal(np.isfinite(got[k]), np.isfinite(r)), k


@pytest.mark.parametrize("L", [1, 24])
@pytest.mark.parametrize("plant", sorted(FINITE))
def test_large_calls_equal_small_ones(data_dir, plant, L):
    """Out-of-range operands in the list form: the bits of calls of 60 columns."""
    b = _batch(_large(), L, FINITE[plant])
    whole = _run(data_dir, b, abi.FP64)
    for c0 in range(0, int(b["ncol"]), 60):
        part = {k: v[c0:c0 + 60] if isinstance(v, np.ndarray) and v.shape[:1] == (int(b["ncol"]),) else v
                for k, v in b.items()}
        part["ncol"] = len(part["acosz"])
        for k, v in _run(data_dir, part, abi.FP64).items():
            assert np.array_equal(v, whole[k][c0:c0 + 60]), k
