"""Objects used from several host threads at once, each on its own stream: filters and
MMA (cooperative kernels that fill the device), and an evaluation with multigrid
solves (dependent launches, a cluster, graphs).  Results equal to the bit those of one
thread alone.
"""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _filter(n, rmin, reps):
    from topopt_in_petsc_transient_gb300 import Filter
    nel = int(np.prod(n))
    x = torch.tensor(np.random.default_rng(nel).random(nel), device="cuda")
    out = torch.zeros(4, nel, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = Filter(*n, 2, rmin)
    for _ in range(reps):
        out[2].copy_(-x ** 3)
        out[3].fill_(1.0 / nel)
        torch.cuda.current_stream().synchronize()
        f.FilterProject(x, out[0], out[1], True, 4.0, 0.5)
        f.Gradients(x, out[0], out[2], 1, out[3], True, 4.0, 0.5)
    return out.cpu().numpy()


def _mma(n, reps):
    from topopt_in_petsc_transient_gb300 import MMA
    rng = np.random.default_rng(n)
    x, df = (torch.tensor(v, device="cuda") for v in (0.2 + 0.6 * rng.random(n), -rng.random(n)))
    dg = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    lo, hi = torch.zeros_like(x), torch.zeros_like(x)
    torch.cuda.synchronize()
    m = MMA(n, 1)
    for _ in range(reps):
        m.SetOuterMovelimit(0.0, 1.0, 0.05, x, lo, hi)
        m.Update(x, df, [float(x.mean()) - 0.4], dg, lo, hi)
    return x.cpu().numpy()


def _evaluate(reps):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    n = (32, 16, 16)
    x = 0.2 + 0.6 * np.random.default_rng(1).random(np.prod(n))
    df = np.zeros(x.size)
    le = LinearElasticity(*n, nlvls=4, ncp=2, tsc=3, t1=6.0, objective=3, loadsignal=0, dalpha=0.0, dbeta=1e-3,
                          mass_precond=0, adaptive_kappa=0.0)
    for _ in range(reps):
        le.CompleteInitialState(x, 1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)
        le.GenerateCheckPoints()
        df[0] = le.ComputeObjectiveSensitivities(df)
    return df


def test_threads(gpu):
    jobs = [lambda: _filter((96, 48, 48), 2.0, 20), lambda: _filter((64, 64, 30), 24.0, 6), lambda: _mma(400000, 10),
            lambda: _evaluate(4), lambda: _evaluate(4)]
    alone = [j() for j in jobs]
    got = [None] * len(jobs)

    def work(i):
        try:
            got[i] = jobs[i]()
        except Exception as e:  # reported below
            got[i] = e
    for _ in range(2):
        ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for i, (a, b) in enumerate(zip(alone, got)):
            assert not isinstance(b, Exception), (i, b)
            assert np.array_equal(a, b), i
