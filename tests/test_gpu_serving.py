"""GPU tests of the serving engine (libops_b200.so, ob2s_*).

* Continuous batching does not change results: a request's solution is
  bit-identical alone and in a mix of other Poisson and ADI requests of
  different sizes that join and leave while it runs.
* Poisson solutions meet the tolerance: the relative residual
  ||b - A x|| / ||b|| recomputed on the CPU (oracle/serving_oracle.py) from
  the fetched solution is at most 1e-8 (x 1.05 for the residual's own
  round-off), in FP64 and in the mixed form.
* Heat requests (backward-Euler steps, each a CG solve): one step meets the
  tolerance against u0 recomputed on the CPU, and several steps agree with
  the same steps solved by a sparse direct solver to the solve accuracy.
* ADI requests match the CPU restatement of the reference's adi step
  (preproc + x/y/z Thomas, z added to u) to 1e-13 of the field's scale
  (same operations in the same order, IEEE without contraction).
"""

import numpy as np
import pytest

from oracle import serving_oracle as so
from ops_b200 import serving

pytestmark = pytest.mark.gpu


def finish_all(eng, iters=8, limit=200000):
    out = {}
    for _ in range(limit):
        for rid in eng.run(iters):
            out[rid] = eng.result(rid)
        if eng.active() == 0:
            return out
    raise AssertionError("requests did not finish")


@pytest.mark.parametrize("mode", [serving.FP64, serving.MIXED])
def test_result_same_alone_and_in_mix(mode):
    eng = serving.Engine(mode)
    try:
        a = eng.submit(serving.POISSON2D, 150, 11)
        finish_all(eng)
        alone = eng.fetch(a, 150 * 150)
        ra = eng.result(a)
        eng.release(a)
        # the same request among others; more join while it runs
        others = [eng.submit(serving.POISSON2D, n, 20 + n) for n in (64, 333, 97)]
        others.append(eng.submit(serving.ADI3D, 40, 7, 4))
        others.append(eng.submit(serving.HEAT2D, 90, 8, 2))
        b = eng.submit(serving.POISSON2D, 150, 11)
        eng.run(5)
        others += [eng.submit(serving.POISSON2D, 211, 5), eng.submit(serving.ADI3D, 33, 9, 3)]
        res = finish_all(eng)
        mixed = eng.fetch(b, 150 * 150)
        rb = eng.result(b)
        assert rb.iterations == ra.iterations and rb.outer == ra.outer
        assert np.array_equal(alone, mixed)
        for rid in [b] + others:
            eng.release(rid)
    finally:
        eng.close()


@pytest.mark.parametrize("mode", [serving.FP64, serving.MIXED])
def test_poisson_meets_tolerance(mode):
    eng = serving.Engine(mode)
    try:
        ids = {eng.submit(serving.POISSON2D, n, 100 + n): n for n in (64, 129, 300)}
        res = finish_all(eng)
        for rid, n in ids.items():
            x = eng.fetch(rid, n * n).reshape(n, n)
            rel = so.relative_residual(x, 100 + n)
            assert rel <= 1.05e-8, (n, rel, res[rid].rel_residual)
            assert abs(rel - res[rid].rel_residual) <= 1e-3 * rel + 1e-15
            eng.release(rid)
    finally:
        eng.close()


def test_engine_made_beside_work_on_the_default_stream():
    """The engine's slots and grid-barrier words are cleared in the order of
    its own stream: an engine made and run while the default stream is busy
    for half a second solves as it does on an idle device."""
    import torch
    sol = []
    for busy in (False, True):
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(1_000_000_000)  # cycles, on the default stream
        eng = serving.Engine(serving.FP64)
        try:
            rid = eng.submit(serving.POISSON2D, 220, 9)
            res = finish_all(eng)[rid]
            assert res.done == 1
            sol.append((eng.fetch(rid, 220 * 220), res.iterations))
            eng.release(rid)
        finally:
            eng.close()
    torch.cuda.synchronize()
    assert sol[0][1] == sol[1][1] and np.array_equal(sol[0][0], sol[1][0])


def test_barrier_that_gives_up_ends_the_engine(monkeypatch):
    """A grid barrier without a single poll gives up in every CTA (as one
    whose wait runs out does): the run returns an error, and so does every
    later run or submission, at once; a request that had finished can still be
    fetched, and the device serves another engine."""
    import time
    monkeypatch.setenv("OB2S_BARRIER_POLLS", "0")
    eng = serving.Engine(serving.FP64)
    try:
        adi = eng.submit(serving.ADI3D, 24, 77, 3)  # no grid barrier in its steps
        finish_all(eng)
        cg = eng.submit(serving.POISSON2D, 700, 1)
        for _ in range(2):
            t = time.perf_counter()
            with pytest.raises(RuntimeError, match="ob2s_run failed"):
                eng.run(100000)
            assert time.perf_counter() - t < 1.0
        with pytest.raises(RuntimeError, match="ob2s_submit failed"):
            eng.submit(serving.ADI3D, 24, 77, 3)
        assert eng.result(cg).done == 0
        u = eng.fetch(adi, 24 ** 3).reshape(24, 24, 24)
        ref = so.adi_steps(24, 77, 3)
        assert np.max(np.abs(u - ref)) <= 1e-13 * np.max(np.abs(ref))
        eng.release(adi)
        eng.release(cg)
    finally:
        eng.close()
    monkeypatch.delenv("OB2S_BARRIER_POLLS")
    eng = serving.Engine(serving.FP64)
    try:
        rid = eng.submit(serving.POISSON2D, 90, 2)
        finish_all(eng)
        assert so.relative_residual(eng.fetch(rid, 90 * 90).reshape(90, 90), 2) <= 1.05e-8
    finally:
        eng.close()


def test_mixed_matches_fp64_solution():
    sol = {}
    for mode in (serving.FP64, serving.MIXED):
        eng = serving.Engine(mode)
        try:
            rid = eng.submit(serving.POISSON2D, 200, 42)
            finish_all(eng)
            sol[mode] = eng.fetch(rid, 200 * 200)
            eng.release(rid)
        finally:
            eng.close()
    d = np.max(np.abs(sol[serving.MIXED] - sol[serving.FP64])) / np.max(np.abs(sol[serving.FP64]))
    # both meet 1e-8 in the residual; the solutions agree to the solve accuracy
    assert d < 1e-6, d


@pytest.mark.parametrize("mode", [serving.FP64, serving.MIXED])
def test_heat_requests(mode):
    eng = serving.Engine(mode)
    try:
        one = eng.submit(serving.HEAT2D, 190, 31, 1)
        three = eng.submit(serving.HEAT2D, 77, 32, 3)
        pois = eng.submit(serving.POISSON2D, 120, 33)
        res = finish_all(eng)
        x = eng.fetch(one, 190 * 190).reshape(190, 190)
        rel = so.heat_relative_residual(x, so.heat_init(190, 31))
        assert rel <= 1.05e-8, (rel, res[one].rel_residual)
        # A >= I, so each step's error is at most its residual (1e-8 of its
        # right-hand side, whose norm never grows): three steps add up to
        # 3e-8 of ||u0|| at most
        u = eng.fetch(three, 77 * 77).reshape(77, 77)
        ref = so.heat_steps(77, 32, 3)
        assert np.linalg.norm(u - ref) <= 3 * 1.05e-8 * np.linalg.norm(so.heat_init(77, 32))
        xp = eng.fetch(pois, 120 * 120).reshape(120, 120)
        assert so.relative_residual(xp, 33) <= 1.05e-8
        for rid in (one, three, pois):
            eng.release(rid)
    finally:
        eng.close()


@pytest.mark.parametrize("mode", [serving.FP64, serving.MIXED])
def test_heat_steps_same_alone_and_in_mix(mode):
    """Heat requests of several time steps, one of them over more tiles than
    there are CTAs, among many small requests (a CTA then advances several
    requests in turn): the norm that each step's residuals are relative to is
    read by every CTA of the request while the quickest of them start the next
    pass.  Bit-identical alone and in the mix, three times over."""
    cases = [(serving.HEAT2D, 700, 3, 4), (serving.HEAT2D, 130, 4, 6), (serving.HEAT2D, 40, 5, 9)]
    eng = serving.Engine(mode)
    try:
        alone = {}
        for kind, n, seed, steps in cases:
            rid = eng.submit(kind, n, seed, steps)
            res = finish_all(eng)[rid]
            alone[n] = (eng.fetch(rid, n * n), res.iterations, res.outer)
            eng.release(rid)
        for _ in range(3):
            small = [eng.submit(serving.POISSON2D, 16 + 3 * k, k) for k in range(40)]
            ids = {eng.submit(*c): c[1] for c in cases}
            small += [eng.submit(serving.HEAT2D, 20 + k, k, 3) for k in range(20)]
            res = finish_all(eng)
            for rid, n in ids.items():
                assert (res[rid].iterations, res[rid].outer) == alone[n][1:], n
                assert np.array_equal(eng.fetch(rid, n * n), alone[n][0]), n
            for rid in small + list(ids):
                eng.release(rid)
    finally:
        eng.close()


@pytest.mark.parametrize("n,steps", [(24, 3), (41, 2), (70, 1)])
def test_adi_matches_oracle(n, steps):
    eng = serving.Engine(serving.MIXED)
    try:
        rid = eng.submit(serving.ADI3D, n, 77, steps)
        res = finish_all(eng)
        assert res[rid].iterations == steps
        u = eng.fetch(rid, n ** 3).reshape(n, n, n)
        ref = so.adi_steps(n, 77, steps)
        assert np.max(np.abs(u - ref)) <= 1e-13 * np.max(np.abs(ref))
        eng.release(rid)
    finally:
        eng.close()


def test_short_serving_run_completes():
    stream = serving.make_stream(40, 200.0, seed=3, pois_n=(64, 256), adi_n=(32, 64), steps=3)
    eng = serving.Engine(serving.MIXED)
    try:
        st = serving.serve(eng, stream, budget_bytes=int(2e9), iters=8)
    finally:
        eng.close()
    assert st["requests"] == 40
    assert st["max_rel_residual"] <= 1e-8
    assert st["p99_s"] >= st["p50_s"] > 0
