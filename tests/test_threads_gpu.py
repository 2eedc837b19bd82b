"""Several host threads, each with a network or an engine of its own, on one GPU.

A kernel's shared-memory limit belongs to the function in the device: calls of
different sizes that run at the same time may not take it from each other. Every
thread's results are the bits that it computes alone.
"""
import threading

import numpy as np
import pytest

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200.engine import Mlp

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Runs the callables at the same time; their results, in order."""
    out, start = [None] * len(jobs), threading.Barrier(len(jobs))

    def work(i):
        start.wait()
        try:
            out[i] = jobs[i]()
        except Exception as e:  # noqa: BLE001 - raised again by the test's thread
            out[i] = e

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for r in out:
        if isinstance(r, Exception):
            raise r
    return out


def _train(width, depth, rows, batch, epochs):
    rng = np.random.default_rng(width)
    x = rng.standard_normal((rows, 20)).astype(np.float32)
    t = rng.standard_normal((rows, 8)).astype(np.float32)
    mask = (0.05 + rng.random((rows, 8))).astype(np.float32)

    def run():
        net = Mlp(20, width, depth, 8, seed=5)
        hist = net.train(x, t, mask, epochs, batch, 1e-3)
        p = net.get_params()
        net.close()
        return np.concatenate([p, np.asarray(hist, np.float32)])
    return run


def test_networks_of_different_sizes():
    jobs = [_train(128, 3, 6400, 64, 20), _train(8, 1, 6400, 64, 40), _train(40, 2, 6400, 64, 30)]
    alone = [j() for j in jobs]
    for a, b in zip(alone, _together(jobs)):
        assert np.array_equal(a, b)


def _engine(lx, ly, sectors, repeats):
    model = pkg.Model(lx=lx, ly=ly, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)
    opts = pkg.RunOpts(samples=4, lanczos_steps=12)

    def run():
        out = []
        with pkg.Engine(model, opts) as eng:
            for _ in range(repeats):
                for nu, nd in sectors:
                    info = eng.sector_prepare(nu, nd)
                    blocks = [(k % lx, k // lx) for k, d in enumerate(info.block_dims) if d > 0][:2]
                    eng.blocks_ftlm_batched(blocks)
                    out += [a for b in blocks for a in eng.block_spectrum(*b, exact=False)[:2]]
                    eng.blocks_exact_batched(blocks)
                    out += [eng.block_spectrum(*b, exact=True)[0] for b in blocks]
        return np.concatenate(out)
    return run


def test_engines_of_different_sizes():
    jobs = [_engine(3, 3, [(3, 4)], 8), _engine(2, 2, [(2, 2), (1, 2)], 300), _engine(4, 2, [(3, 3)], 40)]
    alone = [j() for j in jobs]
    for a, b in zip(alone, _together(jobs)):
        assert np.array_equal(a, b)
