"""Calls that fit a handle's HBM budget by their size keep fitting it: no job
of a device call is larger than the library's limit."""
import numpy as np
import pytest

from mgcm_rt import abi

pytestmark = pytest.mark.gpu

JOB, SLOTS = 32768, 4   # columns per job of a device tracer call at most, jobs in flight


def _tracers(n, L, seed=5):
    """n columns on the device with clear skies and prescribed dust: one ordinary column, repeated."""
    import torch
    lev = 2 * L + 3
    plev = np.geomspace(0.01, 7.0, lev)
    col = dict(plev=plev, pmid=plev, tlev=np.linspace(160.0, 220.0, lev), tmid=np.linspace(160.0, 220.0, lev),
               qh2o=np.full(lev, 1e-4), tauref=np.full(lev + 1, 0.01), acosz=0.5, als=0.2, albi=0.05, pcol=plev[-1],
               detau=np.zeros((17, 7)), cumtauv=np.zeros((17, 7)))
    b = {k: torch.from_numpy(np.asarray(v, dtype=np.float64)).cuda().expand(*((n,) + np.shape(v))).contiguous()
         for k, v in col.items()}
    b.update(ncol=n, L=L, ptrop=0.0008, active_dust=0, cloudon=0,
             sigma=torch.linspace(0.0, 1.0, lev, dtype=torch.float64).cuda(),
             sol=torch.full((7,), 50.0, dtype=torch.float64).cuda())
    return b


@pytest.fixture(scope="module")
def tables(data_dir, tmp_path_factory):
    """The k tables, with Mie tables of one value each: the tracer calls ask for them."""
    import shutil
    from mgcm_rt import data
    d = tmp_path_factory.mktemp("tables")
    for name in data.REQUIRED:
        shutil.copy(data_dir / name, d / name)
    for name, n in ((data.ICE_VIS_FILE, 15 * 20 * 3 * 7), (data.ICE_IR_FILE, 15 * 20 * 3 * 5),
                    ("Dust_vis_wolff2010_JD_12bands.dat", 20 * 3 * 7), ("Dust_ir_wolff2010_JD_12bands.dat", 20 * 3 * 5)):
        (d / name).write_text("0.5\n" * n)
    return d


def _radiation(tables, L, budget=0):
    return abi.Radiation(tables, max_layers=L, precision=abi.FP64, hbm_budget=budget)


def _used(tables, L, call):
    rt = _radiation(tables, L)
    try:
        call(rt)
        return rt.stats()["hbm_used"]
    finally:
        rt.close()


def test_device_tracer_jobs_stay_within_their_limit(tables):
    """The budget of as many jobs as run at once, each of the largest size,
    holds a call of any size."""
    most = _tracers(180000, 1)

    def call(rt, n):
        b = {k: v[:n] if hasattr(v, "shape") and v.shape[0] == 180000 else v for k, v in most.items()}
        out = rt.run_tracers(dict(b, ncol=n), inplace=True)
        assert bool((out["fluxdni"] == out["fluxdni"][0]).all())   # one column, n times
    rt = _radiation(tables, 1, _used(tables, 1, lambda rt: call(rt, SLOTS * JOB)))
    try:
        for n in (SLOTS * JOB, SLOTS * JOB + 1, 147455, 180000):
            call(rt, n)
    finally:
        rt.close()


@pytest.mark.parametrize("before, n", [(15900, 16200), (3300, 3199)])
def test_earlier_calls_do_not_narrow_the_budget(tables, before, n):
    """A call that fits the budget on a new handle fits it after a call that
    was split into other parts: 15,900 x 24 columns run as 2 jobs, 16,200 as 4;
    3,300 as 2, 3,199 as one."""
    b = _tracers(max(before, n), 24)

    def call(rt, m):
        return rt.run_tracers(dict({k: v[:m] if hasattr(v, "shape") and v.shape[0] == b["ncol"] else v
                                    for k, v in b.items()}, ncol=m), inplace=True)
    budget = max(_used(tables, 24, lambda rt: call(rt, before)), _used(tables, 24, lambda rt: call(rt, n)))
    rt = _radiation(tables, 24, budget)
    try:
        want = {k: v.cpu() for k, v in call(rt, before).items()}
        for m in (n, before, n):
            got = call(rt, m)
            assert rt.stats()["hbm_used"] <= budget
            for k, v in want.items():
                assert bool((got[k].cpu()[:1] == v[:1]).all()), k
    finally:
        rt.close()


def test_host_calls_after_one_another(data_dir):
    """The same for host buffers: one job of 3,000 columns, then three of 2,000."""
    from mgcm_rt import synth
    b = synth.make_batch(6000, L=2, seed=8, cloud=False)
    few = {k: v[:3000] if isinstance(v, np.ndarray) and v.shape[0] == 6000 else v for k, v in b.items()}
    few["ncol"] = 3000
    budget = _used(data_dir, 2, lambda rt: rt.run(b))
    rt = _radiation(data_dir, 2, budget)
    try:
        a, c = rt.run(few), rt.run(b)
        assert rt.stats()["hbm_used"] <= budget
        for k, v in a.items():
            assert np.array_equal(v, c[k][:3000]), k
    finally:
        rt.close()


def test_request_after_calls(tables):
    """A budget that holds a call and a request holds them after another call too."""
    import torch
    from mgcm_rt import synth
    t = _tracers(16200, 24)
    b = synth.make_batch(8000, L=24, seed=9, cloud=False)
    b = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v for k, v in b.items()}

    def call(rt, m):
        rt.run_tracers(dict({k: v[:m] if hasattr(v, "shape") and v.shape[0] == 16200 else v for k, v in t.items()},
                            ncol=m), inplace=True)

    def request(rt):
        ticket, out = rt.submit(b)
        rt.wait(ticket, 60.0)
        return {k: v.cpu().numpy() for k, v in out.items()}
    budget = _used(tables, 24, lambda rt: call(rt, 16200)) + _used(tables, 24, request)
    rt = _radiation(tables, 24)
    want = request(rt)
    rt.close()
    rt = _radiation(tables, 24, budget)
    try:
        call(rt, 15900)
        call(rt, 16200)
        for k, v in request(rt).items():
            assert np.array_equal(v, want[k]), k
        call(rt, 15900)
        assert rt.stats()["hbm_used"] <= budget
    finally:
        rt.close()


@pytest.mark.parametrize("L, budget", [(24, 115838464), (48, 213642752), (99, 421348864)])
def test_scratch_of_a_column(data_dir, L, budget):
    """1,000 columns fit the scratch that a column block of plain arrays (no
    padded records) takes with the flux rows of its 204 systems."""
    import torch
    from mgcm_rt import synth
    b = synth.make_batch(1000, L=L, seed=4, cloud=False)
    b = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v for k, v in b.items()}
    rt = _radiation(data_dir, L, budget)
    try:
        ticket, _ = rt.submit(b)
        rt.wait(ticket, 60.0)
    finally:
        rt.close()
