"""Input checks of calls large enough that a CTA of the stage takes four
columns: a bad value in every column of a tile and in the last, partial one, at
inner levels and bands, in every DETAU, and in the grid of fewer layers of a
call over two."""
import numpy as np
import pytest

from mgcm_rt import abi, synth

pytestmark = pytest.mark.gpu


def _device(b):
    import torch
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v for k, v in b.items()}


def _columns():
    import torch
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count + 7   # 3 columns in the last tile


def _status(call, dev, name, index, value=np.nan):
    """The call's status with one value of dev[name] replaced."""
    keep = {n: dev[n].clone() for n in {name, "detau", "cumtauv"}}
    dev[name][index] = value
    try:
        call()
        return 0
    except abi.RTError as e:
        return e.code
    finally:
        for n, v in keep.items():
            dev[n].copy_(v)


@pytest.mark.parametrize("L", [1, 24])
def test_tiles_of_four_columns(data_dir, L):
    n, lev1 = _columns(), 2 * L + 4
    rt = abi.Radiation(data_dir, max_layers=L, precision=abi.FP64)
    dev = _device(synth.make_batch(n, L=L, seed=92, cloud=True, night_frac=0.5))
    out = abi.alloc_outputs(n, L, device=dev["plev"].device)

    def status(*a):
        return _status(lambda: rt.run(dev, out, inplace=True), dev, *a)
    try:
        assert status("als", 0, 0.25) == 0
        for c in [*range(8, 12), *range(n - 3, n)]:
            for name, index in (("pmid", (c, L)), ("tauref", (c, lev1 - 1)), ("gvcld", (c, 3, lev1 // 2)),
                                ("qsidst", (c, 2, lev1 - 1)), ("albi", (c,))):
                assert status(name, index) == -2, (name, index)
            assert status("tlev", (c, lev1 // 2), 49.0) == -3, c
        for k in range(lev1):
            assert status("qxidst", (k % n, k % 5, k)) == -2, k
            assert status("gvdst", (k % n, k % 7, k)) == -2, k
        for q in range(119):
            assert status("detau", (q, q // 7, q % 7)) == -2, q
    finally:
        rt.close()


def test_grids_of_different_layers(data_dir):
    rt = abi.Radiation(data_dir, max_layers=24, precision=abi.FP64)
    grids = [_device(synth.make_batch(_columns(), L=L, seed=93 + L, cloud=True, night_frac=0.5)) for L in (24, 3)]
    outs = [abi.alloc_outputs(int(b["ncol"]), int(b["L"]), device=b["plev"].device) for b in grids]
    try:
        for g, c in ((1, 0), (1, _columns() - 1), (0, _columns() - 1)):
            for name, index in (("plev", (c, 4)), ("taurefcld", (c, 9)), ("qxvdst", (c, 6, 9)), ("detau", (c, 16, 6))):
                assert _status(lambda: rt.run_multi(grids, outs), grids[g], name, index) == -2, (g, name, index)
        rt.run_multi(grids, outs)
    finally:
        rt.close()
