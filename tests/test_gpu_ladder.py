"""The ladder form of PT-ICM (slots spread over CTAs) against the fused form:
the same seed gives the same chain, logs, counts and samples, bit for bit."""
import numpy as np
import pytest

from tamc_b200 import instances as gi

pytestmark = pytest.mark.gpu


def _host(tb, kind):
    name, size = kind.split(":")
    n = int(size)
    if name in ("pm2", "gauss2"):
        h = tb.HostInstance.parse(gi.lattice(n, 2, name[:-1], 3))
    elif name in ("pm3", "gauss3"):
        h = tb.HostInstance.parse(gi.lattice(n, 3, name[:-1], 4))
    elif name == "rrg":
        h = tb.HostInstance.parse(gi.sa_regular(n, 3, 5))
    elif name == "site":
        h = tb.HostInstance.parse("0 0 0.7\n")
    else:
        h = tb.HostInstance.parse(gi.qubo_er(n, 6.0, 6), qubo=True)
    h.add_suscept(np.cos(0.3 * np.arange(h.n)))
    return h


def _everything(r):
    r.sync()
    steps, en, st = r.gs()
    t = r.samples()
    tags, trips, hist = r.round_trips()
    spins, final = r.state()
    return [steps, en, st, r.acceptance(), tags, trips, hist, spins, final, np.array(t.e), np.array(t.q),
            np.array(t.samples), np.array(t.suscept)]


def _same(a, b):
    for x, y in zip(a, b):
        assert x.dtype == y.dtype and x.shape == y.shape and x.tobytes() == y.tobytes()


# kind:size, temperatures, chains, threads, Houdayer moves, sample limiting:
# lattices with and without multi-spin coding (rows of 4 and 6), three-row and
# uneven rows with self-couplings, word remainders and single words, one slot
# to 64, odd chains, both exchange semantics
@pytest.mark.parametrize("kind,nt,C,threads,icm,level", [
    ("pm2:8", 16, 2, 1, True, 0), ("pm2:16", 32, 2, 8, True, 2), ("pm3:6", 33, 2, 8, True, 1),
    ("pm2:5", 7, 4, 1, True, 0), ("gauss2:9", 64, 2, 1, True, 0), ("gauss3:8", 24, 2, 8, True, 1),
    ("rrg:100", 12, 2, 8, True, 0), ("rrg:1030", 9, 3, 1, True, 2), ("qubo:61", 21, 2, 8, True, 0),
    ("qubo:1333", 13, 2, 1, True, 0), ("gauss2:32", 40, 4, 8, True, 0), ("pm2:7", 5, 1, 8, True, 1),
    ("qubo:300", 17, 2, 8, False, 0), ("site:1", 3, 2, 1, True, 0), ("gauss2:4", 1, 2, 8, True, 0),
    ("gauss2:4", 64, 32, 8, True, 2),
])
def test_ladder_and_fused_forms_identical(tb, gpu, monkeypatch, kind, nt, C, threads, icm, level):
    d = gpu.upload(_host(tb, kind))
    b = tb.geometric_betas(0.2, 5.0, nt) if nt > 1 else np.array([0.9], np.float32)
    p = tb.PtParams(60, b, nt // 2, 0.5, icm, C, threads, 7, 9, level)
    got = {}
    for form in ("fused", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        got[form] = _everything(tb.PtRun(d, p, 77).run())
    _same(got["fused"], got["ladder"])


# 3375 and 13824 sites (rows kept in shared memory, and not), against the plain form
@pytest.mark.parametrize("side,kind,nt", [(15, "gauss", 6), (24, "gauss", 5), (24, "pm", 5), (16, "gauss", 64)])
def test_ladder_and_plain_forms_identical_on_large_lattices(tb, gpu, monkeypatch, side, kind, nt):
    h = tb.HostInstance.parse(gi.lattice(side, 3, kind, 8))
    h.add_suscept(gi.fourier_weights(side, 3, 0))
    d = gpu.upload(h)
    p = tb.PtParams(24, tb.geometric_betas(0.2, 5.0, nt), nt // 2, 0.5, True, 2, 8, 5, 5, 0)
    got = {}
    for form in ("plain", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        got[form] = _everything(tb.PtRun(d, p, 5).run())
    _same(got["plain"], got["ladder"])


def test_ladder_runs_in_parts_from_a_given_state(tb, gpu, monkeypatch):
    d = gpu.upload(_host(tb, "gauss2:10"))
    p = tb.PtParams(50, tb.geometric_betas(0.2, 5.0, 10), 4, 0.2, True, 2, 8, 6, 6, 0)
    spins = np.where(np.random.default_rng(1).random((2, 10, 100)) < 0.5, -1, 1).astype(np.int8)
    got = {}
    for form in ("fused", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        r = tb.PtRun(d, p, 9)
        first = r.state()
        r.set_state(spins)
        e0 = r.state()[1]
        r.run(1).run(2)
        mid = r.state()
        got[form] = [*first, e0, *mid, *_everything(r.run(31).run())]
    _same(got["fused"], got["ladder"])


@pytest.mark.parametrize("side,dim,other", [(8, 2, "fused"), (24, 3, "plain")])
def test_ladder_rounds_that_are_given_up_run_in_another_form(tb, gpu, monkeypatch, side, dim, other):
    # a poll limit of zero: the first CTA to wait at a barrier gives up, nothing
    # of those rounds is kept, and the run goes on in the form `other`
    d = gpu.upload(tb.HostInstance.parse(gi.lattice(side, dim, "gauss", 2)))
    p = tb.PtParams(20, tb.geometric_betas(0.2, 5.0, 6), 3, 0.5, True, 2, 8, 5, 5, 0)
    monkeypatch.setenv("TAMC_PT_FORM", other)
    want = _everything(tb.PtRun(d, p, 3).run())
    monkeypatch.setenv("TAMC_PT_FORM", "ladder")
    monkeypatch.setenv("TAMC_LADDER_POLLS", "0")
    _same(want, _everything(tb.PtRun(d, p, 3).run()))


# ladder: several runs a launch, two launches where 296 CTAs of 512 threads are
# resident at once; polls 0: every run's rounds are given up and run fused
@pytest.mark.parametrize("form,threads,polls", [("ladder", "512", None), ("ladder", "128", None), ("", None, None),
                                                ("ladder", "256", "0")])
@pytest.mark.parametrize("how", ["serve", "batch"])
def test_several_runs_in_the_ladder_form_equal_the_fused_form(tb, gpu, monkeypatch, how, form, threads, polls):
    kinds = ["qubo:61", "pm2:12", "gauss3:6", "qubo:300", "rrg:130", "gauss2:9", "pm2:16", "qubo:700", "site:1",
             "pm3:6", "rrg:40", "gauss2:17"]
    if how == "batch":
        kinds = kinds[:4]
    hosts = [_host(tb, k) for k in kinds]
    params = [tb.PtParams(70, tb.geometric_betas(0.2, 5.0, 12 + k), 5, 0.5, True, 2, 8, None, None, 0)
              for k in range(len(kinds))]

    def run():
        if how == "serve":
            srv = tb.Server(gpu, 8 << 30, 64, 25)
            ids = [srv.submit(h, p, 3 + k) for k, (h, p) in enumerate(zip(hosts, params))]
            while any(srv.step()):
                pass
            return [x for i in ids for x in (*srv.state(i), np.float32(srv.result(i)[1]), np.uint32(srv.result(i)[2]))]
        b = tb.Batch(gpu)
        for k, (d, p) in enumerate(zip(gpu.upload_many(hosts), params)):
            b.add(d, p, 3 + k)
        b.run()
        logs = b.gs_all()
        return [x for k in range(len(kinds)) for x in (*b.state(k), b.acceptance(k), *b.round_trips(k), *logs[k])]

    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    want = run()
    monkeypatch.setenv("TAMC_PT_FORM", form)
    if threads:
        monkeypatch.setenv("TAMC_PT_T", threads)
    if polls:
        monkeypatch.setenv("TAMC_LADDER_POLLS", polls)
    _same(want, run())


# serial exchange with few and with most pairs swapping: the fused form walks the
# pairs in the second, the ladder form never does
@pytest.mark.parametrize("nt", [2, 6, 7, 8, 32, 33, 34, 64])
@pytest.mark.parametrize("hi", [0.02, 0.5, 5.0])
def test_serial_exchange_of_ladder_and_fused_forms_identical(tb, gpu, monkeypatch, nt, hi):
    d = gpu.upload(_host(tb, "qubo:61"))
    p = tb.PtParams(80, tb.geometric_betas(0.01, hi, nt), nt // 2, 0.0, True, 2, 1, 7, 9, 0)
    got = {}
    for form in ("fused", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        got[form] = _everything(tb.PtRun(d, p, 5).run())
    _same(got["fused"], got["ladder"])


# couplings beyond the fixed point's range (2^31): sums of them wrap, in every form alike
@pytest.mark.parametrize("value", [3e9, 3e30, np.inf, np.nan])
@pytest.mark.parametrize("kind", ["gauss2:9", "gauss3:6", "rrg:100", "qubo:300"])
@pytest.mark.parametrize("threads,C", [(8, 2), (1, 4)])
def test_ladder_and_other_forms_identical_on_huge_couplings(tb, gpu, monkeypatch, kind, value, threads, C):
    h = _host(tb, kind)
    row_ptr, col, J, bias = h.csr()
    J = np.array(J, np.float32)
    J[np.random.default_rng(2).integers(0, len(J), len(J) // 30 + 1)] = value
    d = gpu.upload(tb.HostInstance.from_csr(row_ptr, col, J, bias))
    p = tb.PtParams(40, tb.geometric_betas(0.01, 2.0, 12), 3, 0.3, True, C, threads, 7, 9, 0)
    got = {}
    for form in ("fused", "plain", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        got[form] = _everything(tb.PtRun(d, p, 9).run())
    _same(got["fused"], got["plain"])
    _same(got["fused"], got["ladder"])
