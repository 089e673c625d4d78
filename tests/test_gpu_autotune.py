"""The launch-shape autotuner (mxg_autotune): it picks, per tunable, one of
its candidates, keeps the choice for the process, and a solve under the chosen
shapes still matches the reference's eigenvalues (the shapes change only the
launch geometry and the order of floating-point sums)."""
import numpy as np
import pytest

import maxwell_gb300 as mx

pytestmark = pytest.mark.gpu


def _solve(g):
    ie, m = int(g["ieigs"]), int(g["m"])
    s = mx.Solver(g["kappa"], n0=int(g["n0"]), L=int(g["L"]), ieigs=ie, m=m, method=1, precision=1,
                  max_nested=40, max_steps=40, wave=len(g["factors"]), relative=0, tol=float(g["tol"]))
    lam, steps, res = s.solve(g["factors"])
    return lam[:, :ie], res[:, :ie]


def test_autotune_choice_and_solve(golden):
    g = golden("eigs_n32_disc.npz")
    default = mx.get_tuning()
    try:
        t = mx.autotune(256, 8, 8, reps=3)
        assert t["gram_waves"] in (1, 2, 4, 8, 16)
        assert t["combine_ctas"] in (1, 2, 3, 4)
        assert t["residual_sites"] in (8, 16, 32, 64, 128)
        assert t["node_strip"] in (0, 64, 128) and t["node_band"] in (4, 8, 16, 32, 64)
        assert t["restrict_strip_log2"] == default["restrict_strip_log2"]   # not searched
        assert mx.get_tuning() == t
        # the extreme shapes too (strips of coarse rows at every level, and at none)
        for shape in ({"gram_waves": 1, "combine_ctas": 1, "residual_sites": 128, "node_strip": 64, "node_band": 1,
                       "restrict_strip_log2": 0},
                      {"gram_waves": 16, "combine_ctas": 4, "residual_sites": 8, "node_strip": 128,
                       "node_band": 64, "restrict_strip_log2": 62}, t):
            mx.set_tuning(**shape)
            lam, res = _solve(g)
            want = g["lam"][:, :int(g["ieigs"])]
            assert np.abs(lam - want).max() / want.max() < 1e-8, shape
            assert res.max() <= float(g["tol"])
    finally:
        mx.set_tuning(**default)


def test_tuning_before_the_first_solve():
    """A node sweep chosen after a solver is made and before its first solve
    takes effect (the launches of that solve are those of a solver made under
    the choice), and stays with the solver's graphs afterwards."""
    default = mx.get_tuning()
    n0, L, m = 8, 4, 4
    kap = np.full((n0 << L) ** 2, 0.5)
    fac = np.exp(1j * np.array([[0.9, 1.7]]))

    def solver():
        return mx.Solver(kap, n0=n0, L=L, ieigs=2, m=m, method=1, precision=1, max_nested=3, max_steps=2, wave=1,
                         relative=1, tol=1e-30)

    def launches(s, **tuning):
        mx.set_tuning(**{**default, **tuning})
        s.solve(fac)
        return s.stats()[1]

    try:
        mx.set_tuning(**default)
        early = solver()
        bands = launches(solver())
        tiled = launches(early, node_strip=64)
        mx.set_tuning(**{**default, "node_strip": 64})
        late = solver()
        assert launches(solver(), node_strip=64) == tiled != bands
        assert launches(late, node_strip=0) == bands
        assert launches(early, node_strip=0) == tiled
    finally:
        mx.set_tuning(**default)


@pytest.mark.parametrize("L, K", [(5, 4), (6, 2)])
def test_autotune_does_not_slow_the_solver(L, K):
    """A solver under the chosen shapes is no slower than under the default
    ones (with a tenth for the timing; a tiled node sweep chosen against the
    row kernels, which these levels no longer run, cost it 28 to 32 %)."""
    import time
    default = mx.get_tuning()
    n0, m = 8, 16
    n = n0 << L
    i = np.arange(n) / n
    X, Y = np.meshgrid(i, i)
    kap = np.where((X - 0.5) ** 2 + (Y - 0.5) ** 2 <= 0.09, 1.0 / 12.0, 1.0).reshape(-1)
    t = np.linspace(0.3, 2.5, K)

    def seconds():
        s = mx.Solver(kap, n0=n0, L=L, ieigs=12, m=m, method=1, precision=1, max_nested=20, nested_tol=1e-2,
                      max_steps=40, wave=K, relative=1, tol=1e-7)
        times = []
        for _ in range(4):
            t0 = time.perf_counter()
            s.solve(np.exp(1j * np.stack([t, 0.4 * t], 1)))
            times.append(time.perf_counter() - t0)
        return min(times[1:])

    try:
        mx.set_tuning(**default)
        before = seconds()
        mx.autotune(n, K, m, 3)
        assert seconds() < 1.1 * before
    finally:
        mx.set_tuning(**default)
