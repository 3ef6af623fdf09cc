"""Two contexts in two host threads, each with solves whose cooperative launches take
different amounts of shared memory: every solution is the lone solve's bit for bit."""
import threading

import numpy as np
import pytest

from dachshund_gb300 import (Context, MixedParams, PCGParams, SignalCovarParams, WFVectorW,
                             pixel_to_wpixel, synth)

pytestmark = pytest.mark.gpu
S = SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA, eval="exact")


def scattered(n):
    rng = np.random.default_rng(n)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, (12.5 * n) ** (1 / 3), (n, 3))
    rec[:, 3] = 1 / rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n)
    return rec


def plain(ctx, n):
    op = WFVectorW(ctx, scattered(n), S)
    return lambda: op.solve_pcg(PCGParams(40, 50, 1e-12))[0]


def mixed(ctx, n):
    op = WFVectorW(ctx, scattered(n), S)
    return lambda: op.solve_mixed(MixedParams(tol=1e-6))[0]


def skewers(ctx, n_sk, n_per):
    w = synth.small(n_sk, n_per, float(np.ceil(2.5 * np.sqrt(n_sk))), seed=3)
    op = WFVectorW(ctx, pixel_to_wpixel(w.pixels), S)
    op.set_cluster_preconditioner(n_sk, n_per, 4, 16)
    op.set_skewer_grid(n_sk, n_per)
    return lambda: op.solve_mixed(MixedParams(tol=1e-8))[0]


def contexts(kind):
    """(make, size) of each thread: plain solves with one CTA per SM and two, mixed
    ones with one row per thread and two, structured ones of short and long skewers."""
    return {"plain": [(plain, (4000,)), (plain, (9000,))],
            "mixed": [(mixed, (3000,)), (mixed, (80000,))],
            "skewers": [(skewers, (40, 40)), (skewers, (60, 240))],
            "all": [(plain, (9000,)), (mixed, (20000,)), (skewers, (60, 240))]}[kind]


@pytest.mark.parametrize("kind", ["plain", "mixed", "skewers", "all"])
def test_contexts_in_threads(kind):
    jobs = contexts(kind)
    ctxs = [Context(0) for _ in jobs]
    solves = [make(c, *size) for c, (make, size) in zip(ctxs, jobs)]
    want = [s() for s in solves]
    start, errors = threading.Barrier(len(jobs)), []

    def loop(k):
        try:
            start.wait()
            for _ in range(12):
                if not np.array_equal(solves[k](), want[k]):
                    errors.append(f"thread {k}: another solution")
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(f"thread {k}: {e!r}")

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    del solves
    for c in ctxs:
        c.close()
    assert not errors, errors
