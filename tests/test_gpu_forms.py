"""Which form of a PT-ICM run and which annealing kernel the comparisons of the
other test files reach, from the lines that TAMC_DEBUG=1 prints: a dispatch rule
that sent them elsewhere would leave those comparing a kernel with itself."""
import re
import threading

import numpy as np
import pytest

import test_gpu_ladder as ladder
import test_gpu_rows as rows
import test_gpu_sa_kernels as sa
from tamc_b200 import instances as gi

pytestmark = pytest.mark.gpu


def _cases(test):
    """The parameter sets of a test of another file."""
    return [m for m in test.pytestmark if m.name == "parametrize"][0].args[1]


def _printed(capfd, pattern):
    return re.findall(pattern, capfd.readouterr().err)


def _forms(capfd):
    return _printed(capfd, r"\[tamc\] PT run .*: (\w+),")


@pytest.fixture(autouse=True)
def _debug(monkeypatch):
    monkeypatch.setenv("TAMC_DEBUG", "1")
    monkeypatch.setenv("TAMC_AUTOTUNE", "0")


@pytest.mark.parametrize("kind,nt,C,threads,icm,level", _cases(ladder.test_ladder_and_fused_forms_identical))
def test_form_of_the_ladder_cases(tb, gpu, monkeypatch, capfd, kind, nt, C, threads, icm, level):
    d = gpu.upload(ladder._host(tb, kind))
    b = tb.geometric_betas(0.2, 5.0, nt) if nt > 1 else np.array([0.9], np.float32)
    p = tb.PtParams(60, b, nt // 2, 0.5, icm, C, threads, 7, 9, level)
    for form in ("fused", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        tb.PtRun(d, p, 77)
    # 64 temperatures on 32 chains: 2048 CTAs of 128 threads are not resident at
    # once (8 to an SM at 64 registers), so the ladder form does not take them
    first, second = _forms(capfd)
    assert first in ("fused", "rows")
    assert (second == "ladder") == (nt * C <= 1184)


@pytest.mark.parametrize("side,kind,nt", _cases(ladder.test_ladder_and_plain_forms_identical_on_large_lattices))
def test_form_of_the_large_lattices(tb, gpu, monkeypatch, capfd, side, kind, nt):
    d = gpu.upload(tb.HostInstance.parse(gi.lattice(side, 3, kind, 8)))
    p = tb.PtParams(24, tb.geometric_betas(0.2, 5.0, nt), nt // 2, 0.5, True, 2, 8, 5, 5, 0)
    for form in ("plain", "ladder"):
        monkeypatch.setenv("TAMC_PT_FORM", form)
        tb.PtRun(d, p, 5)
    assert _forms(capfd) == ["plain", "ladder"]


@pytest.mark.parametrize("side,dim,other", _cases(ladder.test_ladder_rounds_that_are_given_up_run_in_another_form))
def test_rounds_are_given_up(tb, gpu, monkeypatch, capfd, side, dim, other):
    d = gpu.upload(tb.HostInstance.parse(gi.lattice(side, dim, "gauss", 2)))
    p = tb.PtParams(20, tb.geometric_betas(0.2, 5.0, 6), 3, 0.5, True, 2, 8, 5, 5, 0)
    monkeypatch.setenv("TAMC_PT_FORM", "ladder")
    monkeypatch.setenv("TAMC_LADDER_POLLS", "0")
    tb.PtRun(d, p, 3).run().sync()
    err = capfd.readouterr().err
    assert re.findall(r"\[tamc\] PT run .*: (\w+),", err) == ["ladder"]
    assert err.count("[tamc] ladder rounds given up: 1 run(s)") == 1


@pytest.mark.parametrize("how", ["serve", "batch"])
@pytest.mark.parametrize("polls", [None, "0"])
def test_several_runs_take_the_ladder_form(tb, gpu, monkeypatch, capfd, how, polls):
    kinds = ["qubo:61", "pm2:12", "gauss3:6", "qubo:300"]
    monkeypatch.setenv("TAMC_PT_FORM", "ladder")
    monkeypatch.setenv("TAMC_PT_T", "256")
    if polls:
        monkeypatch.setenv("TAMC_LADDER_POLLS", polls)
    hosts = [ladder._host(tb, k) for k in kinds]
    params = [tb.PtParams(70, tb.geometric_betas(0.2, 5.0, 12 + k), 5, 0.5, True, 2, 8) for k in range(len(kinds))]
    if how == "serve":
        srv = tb.Server(gpu, 8 << 30, 64, 25)
        for k, (h, p) in enumerate(zip(hosts, params)):
            srv.submit(h, p, 3 + k)
        srv.step()
    else:
        b = tb.Batch(gpu)
        for k, (d, p) in enumerate(zip(gpu.upload_many(hosts), params)):
            b.add(d, p, 3 + k)
        b.run()
    err = capfd.readouterr().err
    plans = re.findall(r"\[tamc\] plan for (\d+) runs: .* (\d+) in the ladder form", err)
    assert plans[0] == ("4", "4")
    given_up = re.findall(r"\[tamc\] ladder rounds given up: (\d+) run", err)
    assert given_up[:1] == (["4"] if polls else [])


@pytest.mark.parametrize("L,nt,C,threads,icm,lo,level", _cases(rows.test_rows_and_general_path_identical))
def test_form_of_the_lattice_rows(tb, gpu, monkeypatch, capfd, L, nt, C, threads, icm, lo, level):
    d = rows._dev(tb, gpu, L)
    b = tb.geometric_betas(0.2, 5.0, nt) if nt > 1 else np.array([0.9], np.float32)
    p = tb.PtParams(60, b, lo, 0.5, icm, C, threads, 7, 9, level)
    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    for on in ("0", "1"):
        monkeypatch.setenv("TAMC_PT_ROWS", on)
        tb.PtRun(d, p, 11)
    assert _forms(capfd) == ["fused", "rows"]


@pytest.mark.parametrize("kind,size,R", _cases(sa.test_annealing_kernels_identical))
def test_kernel_of_the_annealing_cases(tb, gpu, capfd, kind, size, R):
    h = sa._host(tb, kind, size)
    tb.sa_run(gpu.upload(h), np.linspace(0.1, 6.0, 23).astype(np.float32), R, 1, 5)
    # 0 words, 1 table, 2 slices.  Rows of 4: the table, which at 64 x 64 sites does
    # not fit; rows of 3: the table where the busiest of 148 SMs has ten warps of
    # work (32 sites of the largest class x 4 restarts); uneven rows: slices
    warps = -(-(-(-R // 4)) // 148) * -(-np.bincount(h.coloring()[1]).max() // 32)
    want = {"gauss2": 0 if size == 64 else 1, "rrg": 1 if warps >= 10 else 0}.get(kind, 2)
    assert _printed(capfd, r"\[tamc\] SA tile .*: kernel (\d)") == [str(want)]


def test_plans_ask_the_runtime_once(tb, gpu, capfd):
    # requests of a few sizes, steps of a few rounds: the sizes' occupancies are
    # known after the first plan
    srv = tb.Server(gpu, 8 << 30, 64, 5)
    for k in range(60):
        h = ladder._host(tb, f"qubo:{61 + 37 * (k % 5)}")
        srv.submit(h, tb.PtParams(40, tb.geometric_betas(0.2, 5.0, 12 + k % 3), 5, 0.5, True, 2, 8), k)
    while any(srv.step()):
        pass
    asked = [int(x) for x in _printed(capfd, r"\[tamc\] plan for .* (\d+) occupancy queries")]
    assert len(asked) > 2 and asked[-1] == asked[0]


def test_most_shared_memory_of_the_ladder_form(tb, gpu, monkeypatch, capfd):
    # the longest even ring whose rows (26 bytes a site with everything else) a CTA
    # keeps in shared memory; the next ones keep 10 bytes a site there
    p = tb.PtParams(3, np.array([0.5, 1.0], np.float32), 1, 0.5, True, 2, 8)

    def run(n, form):
        x = np.arange(n)
        rows = np.sort(np.stack([(x - 1) % n, (x + 1) % n], 1), 1)
        h = tb.HostInstance.from_csr(2 * np.arange(n + 1), rows.ravel(), np.ones(2 * n), np.zeros(n))
        monkeypatch.setenv("TAMC_PT_FORM", form)
        return tb.PtRun(gpu.upload(h), p, 3)

    lo, hi = 6000, 14000
    while hi - lo > 2:
        mid = (lo + hi) // 4 * 2
        run(mid, "ladder")
        form, smem = _printed(capfd, r"\[tamc\] PT run .*: (\w+), threads=\d+ smem=(\d+)")[0]
        assert form == "ladder"
        lo, hi = (mid, hi) if int(smem) > 20 * mid else (lo, mid)
    assert lo > 6000 and hi < 14000
    a, b = run(lo, "ladder").run().sync(), run(lo, "plain").run().sync()
    assert a.state()[0].tobytes() == b.state()[0].tobytes() and a.state()[1].tobytes() == b.state()[1].tobytes()


# scratch that cannot be had: the run, the batch and the server's step take another form
@pytest.mark.parametrize("how", ["run", "serve", "batch"])
def test_ladder_scratch_that_cannot_be_had(tb, gpu, monkeypatch, capfd, how):
    hosts = [ladder._host(tb, k) for k in ("qubo:300", "gauss2:9", "gauss3:6", "qubo:61")]
    p = tb.PtParams(70, tb.geometric_betas(0.2, 5.0, 12), 5, 0.5, True, 2, 8)
    monkeypatch.setenv("TAMC_PT_FORM", "ladder")
    got = []
    for scratch in (None, "0"):
        if scratch:
            monkeypatch.setenv("TAMC_LADDER_SCRATCH", scratch)
        if how == "run":
            got.append([x for h in hosts for x in ladder._everything(tb.PtRun(gpu.upload(h), p, 3).run())])
        elif how == "serve":
            srv = tb.Server(gpu, 8 << 30, 64, 25)
            ids = [srv.submit(h, p, 3) for h in hosts]
            while any(srv.step()):
                pass
            got.append([x for i in ids for x in (*srv.state(i), np.float32(srv.result(i)[1]))])
        else:
            b = tb.Batch(gpu)
            for d in gpu.upload_many(hosts):
                b.add(d, p, 3)
            b.run()
            got.append([x for k in range(4) for x in (*b.state(k), b.acceptance(k))])
        err = capfd.readouterr().err
        if how == "run":
            assert set(re.findall(r"\[tamc\] PT run .*: (\w+),", err)) == {"fused" if scratch else "ladder"}
        else:
            assert "ladder form: 4 runs" in err  # planned, and with no scratch not taken
            assert ("[tamc] no memory for the planned ladder form" in err) == bool(scratch)
    ladder._same(*got)


def _serve(tb, gpu, budget, reqs, steps_between=0):
    """The server and the ids of the requests, each submitted `steps_between` steps after the last."""
    srv = tb.Server(gpu, budget, 64, 10)
    ids = []
    for k, (h, p) in enumerate(reqs):
        for _ in range(steps_between if k else 0):
            srv.step()
        ids.append(srv.submit(h, p, 3 + k))
    return srv, ids


def _footprint(tb, gpu, h, p):
    """The smallest budget that a request is accepted with."""
    lo, hi = 0, 1 << 28
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            tb.Server(gpu, mid, 4, 10).submit(h, p, 1)
            hi = mid
        except tb.TamcError as e:
            assert e.code == -9
            lo = mid
    return hi


# rows of uneven length (sliced rows and scratch) and of one length (scratch alone)
@pytest.mark.parametrize("kind", ["qubo:700", "gauss3:8"])
def test_server_budget_covers_the_ladder_form(tb, gpu, monkeypatch, capfd, kind):
    monkeypatch.setenv("TAMC_PT_FORM", "ladder")
    h = ladder._host(tb, kind)
    p = tb.PtParams(60, tb.geometric_betas(0.2, 5.0, 16), 5, 0.5, True, 2, 8)
    own = _footprint(tb, gpu, h, p)

    def planned():
        """(runs, those in the ladder form) of the last step's plan."""
        found = _printed(capfd, r"\[tamc\] plan for (\d+) runs: .* (\d+) in the ladder form")
        return tuple(int(x) for x in found[-1])

    def results(srv, ids):
        while any(srv.step()):
            pass
        return [x for i in ids for x in (*srv.state(i), np.float32(srv.result(i)[1]))]

    # room for nothing but the footprint: fused, and the second request waits
    srv, ids = _serve(tb, gpu, own, [(h, p), (h, p)])
    assert srv.step() == (1, 1) and planned() == (1, 0)
    got = results(srv, ids)
    # room for both with all they need
    srv, ids = _serve(tb, gpu, 4 * own, [(h, p), (h, p)])
    assert srv.step() == (2, 0) and planned() == (2, 2)
    ladder._same(results(srv, ids), got)
    # room for two footprints: the first request has more until the second needs it
    srv, ids = _serve(tb, gpu, 2 * own, [(h, p), (h, p)], steps_between=2)
    assert planned() == (1, 1)
    assert srv.step() == (2, 0) and planned() == (2, 0)
    ladder._same(results(srv, ids), got)


# rounds in the ladder form, then beside many other runs in the fused form, then in the ladder form again
@pytest.mark.parametrize("kind,nt", [("qubo:300", 24), ("gauss2:17", 32), ("pm3:10", 32)])
def test_rounds_beside_other_runs(tb, gpu, monkeypatch, capfd, kind, nt):
    d = gpu.upload(ladder._host(tb, kind))
    p = tb.PtParams(60, tb.geometric_betas(0.2, 5.0, nt), nt // 3, 0.2, True, 2, 8, 7, 9, 0)
    r = tb.PtRun(d, p, 11).run(20)
    monkeypatch.setenv("TAMC_PT_BESIDE", "1000")
    r.run(45)
    monkeypatch.delenv("TAMC_PT_BESIDE")
    got = ladder._everything(r.run())
    err = capfd.readouterr().err
    assert re.findall(r"\[tamc\] PT run .*: (\w+),", err) == ["ladder"]
    assert re.findall(r"\[tamc\] rounds (\d+) to (\d+) in the fused form beside 1000 contexts", err) == [("20", "45")]
    monkeypatch.setenv("TAMC_PT_FORM", "fused")
    ladder._same(ladder._everything(tb.PtRun(d, p, 11).run()), got)


def test_several_contexts_at_once(tb, gpu):
    """Single runs in the ladder form, a batch and a server on contexts of their own,
    each in a thread, against the same work one after another."""
    kinds = ["qubo:300", "gauss3:8", "rrg:130", "gauss2:17"]
    p = tb.PtParams(300, tb.geometric_betas(0.2, 5.0, 16), 5, 0.5, True, 2, 8)

    def single(kind):
        def work(g):
            return ladder._everything(tb.PtRun(g.upload(ladder._host(tb, kind)), p, 3).run())
        return work

    def batch(g):
        b = tb.Batch(g)
        for d in g.upload_many([ladder._host(tb, k) for k in kinds + ["pm2:16", "pm2:12"]]):
            b.add(d, p, 3)
        b.run()
        return [x for k in range(6) for x in b.state(k)]

    def serve(g):
        srv = tb.Server(g, 8 << 30, 64, 60)
        ids = [srv.submit(ladder._host(tb, k), p, 3) for k in kinds]
        while any(srv.step()):
            pass
        return [x for i in ids for x in srv.state(i)]

    work = [single(k) for k in kinds] * 2 + [batch, serve]
    want = [w(gpu) for w in work]
    got = [None] * len(work)

    def thread(k, g):
        got[k] = work[k](g)

    contexts = [tb.Gpu(0) for _ in work]
    threads = [threading.Thread(target=thread, args=(k, g)) for k, g in enumerate(contexts)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(want, got):
        ladder._same(a, b)


# many restarts on an SM and few sites a class or padded slices, 3-regular instances
# whose CTAs do not fit beside one another: words (0), else table (1) and slices (2)
@pytest.mark.parametrize("kind,size,R,kernel", [
    ("gauss2", 4, 2368, 1), ("gauss2", 4, 2372, 0), ("gauss2", 8, 16384, 1), ("rrg", 2000, 2048, 1),
    ("rrg", 2000, 4096, 0), ("rrg", 2000, 16384, 1), ("rrg", 2400, 1024, 1), ("rrg", 2400, 2048, 0),
    ("rrg", 2600, 592, 1), ("rrg", 2600, 600, 0), ("qubo", 30, 2368, 2), ("qubo", 30, 2372, 0),
    ("qubo", 1000, 8192, 2),
])
def test_annealing_kernel_for_many_restarts(tb, gpu, capfd, kind, size, R, kernel):
    tb.sa_run(gpu.upload(sa._host(tb, kind, size)), np.linspace(0.1, 2.0, 8).astype(np.float32), R, 1, 5)
    assert _printed(capfd, r"\[tamc\] SA tile .*: kernel (\d)") == [str(kernel)]


@pytest.mark.parametrize("kind,kernel", [("gauss2", 1), ("qubo", 2)])
def test_annealing_kernel_of_few_sweeps(tb, gpu, monkeypatch, capfd, kind, kernel):
    d = gpu.upload(sa._host(tb, kind, 30))
    got = []
    for nbeta in (0, 3, 4, 4):
        if len(got) == 3:
            monkeypatch.setenv("TAMC_SA_KERNEL", "words")
        got.append(tb.sa_run(d, np.linspace(0.1, 6.0, nbeta).astype(np.float32), 40, 1, 5))
    # (the words kernel's tile is printed when it is chosen, at the first call)
    assert _printed(capfd, r"\[tamc\] SA tile .*: kernel (\d)") == ["0", str(kernel)]
    assert got[2][0].tobytes() == got[3][0].tobytes() and got[2][1].tobytes() == got[3][1].tobytes()
