"""The annealing kernels for rows of 3 or 4 entries (fields from a table) and
for uneven rows (slices) against the one for any rows: the same seed gives the
same states and energies, bit for bit."""
import numpy as np
import pytest

from tamc_b200 import instances as gi

pytestmark = pytest.mark.gpu


def _host(tb, kind, n):
    if kind == "gauss2":
        return tb.HostInstance.parse(gi.lattice(n, 2, "gauss", 3))
    if kind == "rrg":
        return tb.HostInstance.parse(gi.sa_regular(n, 3, 5))
    if kind == "dense":
        rng = np.random.default_rng(1)
        return tb.HostInstance.parse(gi.to_text(n, [(i, j, rng.standard_normal()) for i in range(n) for j in range(i)]))
    return tb.HostInstance.parse(gi.qubo_er(n, min(9.0, n / 2 - 0.5), 6), qubo=True)


# kind, size, restarts: rows of 4 (table whole, table halved, no room for it),
# rows of 3 (few and many warps of work), uneven rows (single slices, padded
# ones, rows in shared memory and in L2, one class a site), restarts that
# leave quads and words part empty, 4 to 16 restarts a CTA
@pytest.mark.parametrize("kind,size,R", [
    ("gauss2", 3, 1), ("gauss2", 8, 33), ("gauss2", 13, 700), ("gauss2", 40, 601), ("gauss2", 48, 1500),
    ("gauss2", 64, 130), ("rrg", 1000, 515), ("rrg", 2000, 1024), ("rrg", 2402, 604), ("rrg", 30, 2000),
    ("qubo", 3, 2), ("qubo", 7, 5), ("qubo", 251, 100), ("qubo", 333, 2047), ("qubo", 2000, 700), ("qubo", 9000, 37),
    ("dense", 40, 9),
])
def test_annealing_kernels_identical(tb, gpu, monkeypatch, kind, size, R):
    d = gpu.upload(_host(tb, kind, size))
    monkeypatch.setenv("TAMC_AUTOTUNE", "0")
    for nbeta in (0, 1, 23):
        b = np.linspace(0.1, 6.0, nbeta).astype(np.float32)
        e, s = tb.sa_run(d, b, R, 1, 5)
        with monkeypatch.context() as m:
            m.setenv("TAMC_SA_KERNEL", "words")
            e0, s0 = tb.sa_run(d, b, R, 1, 5)
        assert e.tobytes() == e0.tobytes() and s.tobytes() == s0.tobytes()
