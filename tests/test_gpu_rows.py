"""+-J square lattices of even side on lattice rows against the fused kernel's
general path: the same seed gives the same chain, logs, counts and samples, bit
for bit."""
import numpy as np
import pytest

from tamc_b200 import instances as gi
from test_gpu_ladder import _everything, _same

pytestmark = pytest.mark.gpu


def _dev(tb, gpu, L):
    h = tb.HostInstance.parse(gi.lattice(L, 2, "pm", 3 + L))
    h.add_suscept(np.cos(0.3 * np.arange(h.n)))
    return gpu.upload(h)


# side (rows of 8, 16 and 32 lanes, filled and not; sites that leave a chunk of 32
# part empty), temperatures (one to two words), chains (a word or a pair alone, two
# pairs), threads (exchange semantics), Houdayer moves from which slot, sampling
@pytest.mark.parametrize("L,nt,C,threads,icm,lo,level", [
    (4, 1, 1, 8, False, 0, 0), (4, 5, 2, 1, True, 0, 0), (6, 8, 2, 8, True, 3, 1), (8, 32, 2, 8, True, 16, 0),
    (10, 13, 4, 1, True, 12, 2), (12, 33, 2, 8, True, 31, 0), (14, 17, 2, 8, True, 16, 1), (16, 32, 4, 8, True, 0, 0),
    (16, 64, 1, 1, True, 20, 0), (18, 9, 2, 8, False, 2, 2), (24, 40, 2, 1, True, 33, 0), (30, 24, 2, 8, True, 12, 1),
    (32, 32, 2, 8, True, 16, 0), (32, 64, 2, 8, True, 30, 2), (32, 3, 4, 8, True, 1, 0),
])
def test_rows_and_general_path_identical(tb, gpu, monkeypatch, L, nt, C, threads, icm, lo, level):
    d = _dev(tb, gpu, L)
    b = tb.geometric_betas(0.2, 5.0, nt) if nt > 1 else np.array([0.9], np.float32)
    p = tb.PtParams(60, b, lo, 0.5, icm, C, threads, 7, 9, level)
    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    monkeypatch.setenv("TAMC_AUTOTUNE", "0")
    got = {}
    for rows in ("0", "1"):
        monkeypatch.setenv("TAMC_PT_ROWS", rows)
        a = _everything(tb.PtRun(d, p, 11).run())
        r = tb.PtRun(d, p, 11)
        spins, _ = r.state()
        r.set_state(-spins)  # energies from given spins
        got[rows] = a + _everything(r.run())
    _same(got["0"], got["1"])


# a launch of rows alone and one with other runs in it, at each CTA size
@pytest.mark.parametrize("threads", ["128", "256", "512"])
@pytest.mark.parametrize("other", [False, True])
def test_rows_in_a_batch(tb, gpu, monkeypatch, threads, other):
    jobs = [(_dev(tb, gpu, L), nt) for L, nt in ((8, 16), (32, 32), (12, 24), (16, 40))]
    if other:
        jobs.insert(1, (gpu.upload(tb.HostInstance.parse(gi.lattice(9, 2, "gauss", 3))), 12))
    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    monkeypatch.setenv("TAMC_AUTOTUNE", "0")
    got = []
    for rows, T in (("0", "512"), ("1", threads)):
        monkeypatch.setenv("TAMC_PT_ROWS", rows)
        monkeypatch.setenv("TAMC_PT_T", T)
        b = tb.Batch(gpu)
        for k, (d, nt) in enumerate(jobs):
            b.add(d, tb.PtParams(150, tb.geometric_betas(0.2, 5.0, nt), nt // 2, 0.5, True, 2, 8, None, None, 0), 5 + k)
        b.run()
        logs = b.gs_all()
        got.append([x for k in range(len(jobs)) for x in (*b.state(k), b.acceptance(k), *b.round_trips(k), *logs[k])])
    _same(*got)


# the rows' cluster growth against the union-find search, which runs on the general path
@pytest.mark.parametrize("L,nt,C", [(4, 5, 2), (10, 13, 4), (16, 32, 2), (30, 24, 2), (32, 64, 2)])
def test_rows_and_union_find_identical(tb, gpu, monkeypatch, capfd, L, nt, C):
    d = _dev(tb, gpu, L)
    p = tb.PtParams(60, tb.geometric_betas(0.2, 5.0, nt), nt // 3, 0.5, True, C, 8, 7, 9, 0)
    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    monkeypatch.setenv("TAMC_AUTOTUNE", "0")
    monkeypatch.setenv("TAMC_DEBUG", "1")
    got = [_everything(tb.PtRun(d, p, 11).run())]
    monkeypatch.setenv("TAMC_ICM", "uf")
    got.append(_everything(tb.PtRun(d, p, 11).run()))
    err = capfd.readouterr().err
    assert [x for x in ("rows", "fused", "plain", "ladder") if f": {x}, threads" in err] == ["rows", "fused"]
    _same(*got)
