"""Kernels at the sizes where they can go wrong: tile edges, remainders, many contexts at once."""
import math

import numpy as np
import pytest

from helpers import oparams, source

pytestmark = pytest.mark.gpu


def test_ensemble_of_developed_members_matches_members_alone(engine):
    """Sixteen developed displacements whose kernels fill the GPU together end with the bits they
    have alone: no block may read a cell (the pinned one) that another block of its launch writes,
    since blocks start late when other members hold the SMs."""
    E = engine
    import torch

    def member(k):
        N = 128 * (1 + k % 4)
        P = E.default_params(N, N, stype=1, hmtype=4, nu=1.0, diffusion=1, alpha_l=1e-3, alpha_t=1e-4, eps=1e-8,
                             para_eps=1e-10, max_cycles=200, precision=1)
        ctx = E.Context(P)
        i = np.arange(N)
        r = np.hypot(i[:, None], i[None, :])
        c = np.zeros((N + 4, N + 4))
        c[2:-2, 2:-2] = 1.0 / (1.0 + np.exp((r - 0.35 * math.sqrt(2.0) * N) / 3.0))
        ctx.upload(c, source(oparams(P)), ghost=2)
        ctx.set_time(0.0)
        return ctx

    def state(ctx):
        N = ctx.P.N1
        c, p = np.zeros((N + 4, N + 4)), np.zeros((N + 4, N + 4))
        ctx.download(c, p, None, ghost=2)
        return c, p
    alone = []
    for k in range(16):
        ctx = member(k)
        ctx.step()
        alone.append(state(ctx))
        ctx.close()
    for _ in range(3):
        ens = E.Ensemble([member(k) for k in range(16)])
        ens.step(1)
        torch.cuda.synchronize()
        for ctx, (c, p) in zip(ens.members, alone):
            ce, pe = state(ctx)
            assert np.array_equal(ce, c) and np.array_equal(pe, p)
        ens.close()
