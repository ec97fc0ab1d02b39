"""Reference-order mode at the edges of its block-wise kernels, against the CPU
oracle bit for bit: sites around multiples of 32 and 64, rows of uneven length
with self-couplings, chains whose neighbours lie in the same block, one to
more than 64 temperatures, hot and cold ladders, both exchange semantics."""
import numpy as np
import pytest

from tamc_b200 import instances as gi

pytestmark = pytest.mark.gpu


def _text(kind, n):
    if kind == "ring":  # every site's neighbours are the sites beside it
        rng = np.random.default_rng(n)
        e = [(i, i + 1, rng.standard_normal()) for i in range(n - 1)] + [(0, n - 1, 0.5)]
        return gi.to_text(n, e, biases=0.2 * rng.standard_normal(n)), False
    if kind == "rrg":
        return gi.sa_regular(n, 3, n), False
    if kind == "qubo":
        return gi.qubo_er(n, 6.0, n), True
    return gi.lattice(n, 2, "pm", n), False


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("kind,n,nt,C,lo,hi,sweeps", [
    ("ring", 31, 3, 2, 0.1, 2.0, 40), ("ring", 32, 2, 2, 0.1, 2.0, 40), ("ring", 33, 5, 3, 0.1, 5.0, 40),
    ("ring", 65, 1, 2, 0.7, 0.7, 40), ("ring", 64, 70, 2, 0.01, 8.0, 15), ("rrg", 130, 33, 2, 0.2, 5.0, 15),
    ("qubo", 63, 4, 4, 0.02, 1.0, 30), ("qubo", 97, 9, 2, 0.1, 5.0, 30), ("pm", 12, 34, 2, 0.0, 5.0, 12),
    ("pm", 16, 6, 2, 0.2, 5.0, 30),
])
def test_ref_blocks_match_oracle(tb, po, gpu, threads, kind, n, nt, C, lo, hi, sweeps):
    text, qubo = _text(kind, n)
    b = np.linspace(lo, hi, nt).astype(np.float32)
    orc = po.PtRun(po.Instance.from_text(text, qubo=qubo), b, sweeps, 0.3, nt // 2, True, C, threads, sample=4,
                   sample_states=5, sample_limiting=0, seed=n + nt)
    orc.run()
    p = tb.PtParams(sweeps, b, nt // 2, 0.3, True, C, threads, 4, 5, 0)
    run = tb.PtRun(gpu.upload(tb.HostInstance.parse(text, qubo=qubo)), p, n + nt, tb.MODE_REF).run().sync()
    S0, E0, _ = orc.states()
    S1, E1 = run.state()
    assert np.array_equal(S0, S1) and np.array_equal(_bits(E0), _bits(E1))
    assert np.array_equal(orc.acceptance().sum(0), run.acceptance())
    steps, en, _ = run.gs()
    assert [g[0] for g in orc.gs()] == list(steps)
    assert np.array_equal(_bits([g[1] for g in orc.gs()]), _bits(en))


def _matches_oracle(tb, po, gpu, text, qubo, b, C, threads, sweeps, seed):
    nt = len(b)
    orc = po.PtRun(po.Instance.from_text(text, qubo=qubo), b, sweeps, 0.3, nt // 2, True, C, threads, sample=4,
                   sample_states=5, sample_limiting=0, seed=seed)
    orc.run()
    p = tb.PtParams(sweeps, b, nt // 2, 0.3, True, C, threads, 4, 5, 0)
    run = tb.PtRun(gpu.upload(tb.HostInstance.parse(text, qubo=qubo)), p, seed, tb.MODE_REF).run().sync()
    S0, E0, _ = orc.states()
    S1, E1 = run.state()
    assert np.array_equal(S0, S1) and np.array_equal(_bits(E0), _bits(E1))
    assert np.array_equal(orc.acceptance().sum(0), run.acceptance())
    steps, en, _ = run.gs()
    assert [g[0] for g in orc.gs()] == list(steps)
    assert np.array_equal(_bits([g[1] for g in orc.gs()]), _bits(en))


# What stays outside shared memory: the rows (bits, queue and row terms of a
# Houdayer move, and the ladder's exchange state fit: 10 bytes a site and 17 a
# temperature), or everything (the kernels of one thread per stream)
@pytest.mark.parametrize("outside", ["rows", "all"])
@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("kind,n,nt,C,lo,hi,sweeps", [
    ("ring", 33, 5, 3, 0.1, 5.0, 40), ("rrg", 130, 33, 2, 0.2, 5.0, 15), ("qubo", 97, 9, 2, 0.1, 5.0, 30),
    ("pm", 16, 6, 2, 0.2, 5.0, 30),
])
def test_ref_kernels_outside_shared_memory_match_oracle(tb, po, gpu, monkeypatch, outside, threads, kind, n, nt, C, lo,
                                                        hi, sweeps):
    text, qubo = _text(kind, n)
    sites = n * n if kind == "pm" else n
    monkeypatch.setenv("TAMC_REF_SMEM", "0" if outside == "all" else str(10 * sites + 17 * nt + 256))
    _matches_oracle(tb, po, gpu, text, qubo, np.linspace(lo, hi, nt).astype(np.float32), C, threads, sweeps, n + nt)


# energies in one and two passes over the sites; and rows of 229 KB, more than an
# SM's shared memory
@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("kind,n", [("ring", 1024), ("ring", 1025), ("rrg", 2050), ("gauss3", 16)])
def test_ref_large_instances_match_oracle(tb, po, gpu, threads, kind, n):
    text, qubo = (gi.lattice(n, 3, "gauss", n), False) if kind == "gauss3" else _text(kind, n)
    b = np.linspace(0.2, 3.0, 3).astype(np.float32)
    _matches_oracle(tb, po, gpu, text, qubo, b, 2, threads, 6, n)
