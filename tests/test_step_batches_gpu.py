"""The step at the batch sizes where its kernels change form, against the FP64 oracle.

Each row crosses a line of the dispatch: vectors interleaved by 1, 2, 4 or 8
instances with a partial last group (3, 5, 9), the V'p product with 4 x 4 sums
per thread (64 and more), one to four layer rows per thread of the kernel
that applies Hx^T, the preconditioner in one cluster kernel (up to 6 instances of the 30 m
system), in three kernels, and with several layers per CTA (25 instances: 150
(layer, instance) planes for 148 SMs); the cluster kernel for the vector part of
an unpreconditioned iteration with 4 elements per thread (8 m, the fits) and 8
(30 m without its preconditioner), and the separate kernels where the vector does
not fit a cluster (39 m without it).

Tolerances, as in test_tomo_gpu.py and test_fit_gpu.py (relative L2): operators
5e-5, layers after the solve 2e-3, commands 1e-4; six iterations, so that
rounding is not amplified beyond what those tests allow 30.
"""
import dataclasses

import numpy as np
import pytest

from oracle.recon_oracle import SparseFitOracle, TomoOracle, fit_solve, tomo_solve

pytestmark = pytest.mark.gpu

OP_TOL, LAYER_TOL, DM_TOL, ITERS = 5e-5, 2e-3, 1e-4, 6


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b))


def system(name):
    """The preset, or (..._cg) the same tables without the preconditioner; with its assembled fit."""
    from conftest import get_fit_assembled, get_system
    base = name.removesuffix("_cg")
    s = get_system(base)
    if name != base:
        s = dataclasses.replace(s, fdpcg=None, cfg=dataclasses.replace(s.cfg, tomo_precond=0))
    return s, get_fit_assembled(base)


@pytest.mark.parametrize("name,nb", [("scao_8m", 1), ("scao_8m", 9), ("ltao_8m", 3), ("ltao_8m", 5), ("ltao_8m", 65),
                                     ("mcao_30m", 3), ("mcao_30m", 9), ("mcao_30m", 25), ("mcao_30m_cg", 2),
                                     ("elt_39m_cg", 2)])
def test_step_at_batch(name, nb):
    from maos_b200.recon import Reconstructor
    s, fs = system(name)
    to, fo = TomoOracle(s), SparseFitOracle(s, fs)
    rng = np.random.default_rng(100 + nb)
    g = rng.standard_normal((nb, s.ngrad)) * 1e-6
    x = rng.standard_normal((nb, s.nx_total)) * 1e-7
    a = rng.standard_normal((nb, fs.nact)) * 1e-7
    R = Reconstructor(s, nbatch=nb, fit=fs, maxit=ITERS)
    try:
        got = R.apply_L(x), R.apply_R(g), R.apply_fit_L(a)
        R.reset()
        layers, _ = R.tomo(g)
        commands, _ = R.fit()
    finally:
        R.close()
    for b in sorted({0, nb // 2, nb - 1}):
        assert rel(got[0][b], to.tomo_L(x[b])) < OP_TOL
        assert rel(got[1][b], to.tomo_R(g[b])) < OP_TOL
        assert rel(got[2][b], fo.fit_L(a[b])) < OP_TOL
        want, _ = tomo_solve(to, g[b], maxit=ITERS)
        assert rel(layers[b], want) < LAYER_TOL
        assert rel(commands[b], fit_solve(fo, want)[0]) < DM_TOL
