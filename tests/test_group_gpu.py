"""Uneven instances advanced together (mb_group_*).

Three reconstructors of different geometries and batch sizes -- 8 m SCAO
(2 instances), 8 m LTAO (plain CG, 2 instances) and 30 m MCAO (FDPCG,
3 instances) -- are stepped by one group graph in which the tomography
operators are single launches over all their instances.  Every instance's DM
commands must equal those of its own reconstructor stepped alone, bit for bit
(the group runs each member's own arithmetic), over two warm-started steps;
and the group step must take fewer kernel launches than the three steps
alone.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MEMBERS = (("scao_8m", 2), ("ltao_8m", 2), ("mcao_30m", 3))


@pytest.fixture(scope="module")
def group():
    from conftest import get_fit_assembled, get_system
    from maos_b200 import turbulence
    from maos_b200.recon import Reconstructor, ReconGroup
    rs, grads = [], []
    for name, nb in MEMBERS:
        s = get_system(name)
        R = Reconstructor(s, nbatch=nb, fit=get_fit_assembled(name))
        rs.append(R)
        fr = turbulence.gradient_frames(s, seed=3, nframe=2 * nb).astype(np.float32)
        grads.append(torch.tensor(fr.reshape(2, nb, -1), device="cuda"))
    G = ReconGroup(rs)
    yield rs, G, grads
    G.close()
    for R in rs:
        R.close()


def _commands(rs):
    torch.cuda.synchronize()
    return [R.fit_solution().cpu().numpy().copy() for R in rs]


def test_group_step_equals_members_alone(group):
    rs, G, grads = group
    lib = rs[0].lib
    alone = []
    lib.mb_kernel_launches(1)
    for R in rs:
        R.reset()
    for step in range(2):
        for R, g in zip(rs, grads):
            R.step_device(g[step].data_ptr())
        alone.append(_commands(rs))
    n_alone = lib.mb_kernel_launches(1) / 2
    together = []
    for R in rs:
        R.reset()
    for step in range(2):
        G.step_device([g[step].data_ptr() for g in grads])
        together.append(_commands(rs))
    n_group = lib.mb_kernel_launches(1) / 2
    for step in range(2):
        for i, (name, nb) in enumerate(MEMBERS):
            a, b = alone[step][i], together[step][i]
            assert a.shape == (nb, rs[i].nact)
            assert np.all(np.isfinite(b)) and np.abs(a).max() > 0
            assert np.array_equal(a, b), (name, step, float(np.abs(a - b).max()))
    assert G.graph_kernels == n_group
    assert n_group < n_alone, (n_group, n_alone)
    print(f"kernel launches per step: group {n_group:.0f}, members alone {n_alone:.0f}")


def test_group_follows_a_member_table_update(group):
    """After a member's tables change (here a re-autotune, which recaptures
    the member's graph), the group recaptures before its next step and still
    matches the member alone."""
    rs, G, grads = group
    rs[2].autotune(reps=3)
    for R in rs:
        R.reset()
    G.step_device([g[0].data_ptr() for g in grads])
    together = _commands(rs)
    for R in rs:
        R.reset()
    for R, g in zip(rs, grads):
        R.step_device(g[0].data_ptr())
    alone = _commands(rs)
    for i in range(len(rs)):
        assert np.array_equal(alone[i], together[i])


def test_one_launch_per_operator_whatever_the_rows_per_thread():
    """Members whose layer kernels keep 1 (2 instances of the 8 m system), 2 and
    4 layer rows per thread (6 and 23 of the 30 m one) share one launch of it:
    bit for bit the members' own results, and for every application of an
    operator (the right-hand side, A x, A p of each iteration) one launch of
    each kernel instead of one per member."""
    from conftest import get_fit_assembled, get_system
    from maos_b200.recon import Reconstructor, ReconGroup
    rng = np.random.default_rng(22)
    iters, members = 3, (("scao_8m", 2), ("mcao_30m", 6), ("mcao_30m", 23))
    rs, gs, pos = [], [], set()
    try:
        for name, nb in members:
            s = get_system(name)
            pos.add(round(s.wfs[0].dsa / s.pmap.dx))
            rs.append(Reconstructor(s, nbatch=nb, maxit=iters, fit=get_fit_assembled(name)))
            gs.append(torch.as_tensor(rng.standard_normal((nb, s.ngrad)) * 1e-6, dtype=torch.float32, device="cuda"))
        lib = rs[0].lib
        lib.mb_kernel_launches(1)
        for R, g in zip(rs, gs):
            R.step_device(g.data_ptr())
        n_alone, want = lib.mb_kernel_launches(1), _commands(rs)
        G = ReconGroup(rs)
        try:
            for R in rs:
                R.reset()
            G.step_device([g.data_ptr() for g in gs])
            for a, b in zip(_commands(rs), want):
                assert np.array_equal(a, b)
            saved = (len(rs) - len(pos)) + (len(rs) - 1)  # k_pupil_rows: a launch per subaperture/pupil ratio
            assert G.graph_kernels == n_alone - (iters + 2) * saved
        finally:
            G.close()
    finally:
        for R in rs:
            R.close()


def test_a_smaller_system_built_later_leaves_the_larger_usable():
    """The dynamic shared memory a kernel may take belongs to the kernel, which
    every reconstructor shares.  A 39 m system's layer transforms take nearly
    twice what a 30 m one's do: built after it, the 30 m one must not take the
    39 m one's away, in either form of the preconditioner, nor in a group of
    both."""
    from conftest import get_fit_assembled, get_system
    from maos_b200.recon import Reconstructor, ReconGroup
    rng = np.random.default_rng(21)
    rs, gs = [], []

    def alone(i, mode):
        assert rs[i].fdpcg_mode(mode) == mode  # captures the step again
        rs[i].reset()
        rs[i].step_device(gs[i].data_ptr())
        return _commands([rs[i]])[0]

    try:
        for name in ("elt_39m", "mcao_30m"):
            s = get_system(name)
            rs.append(Reconstructor(s, nbatch=1, maxit=3, fit=get_fit_assembled(name)))
            gs.append(torch.as_tensor(rng.standard_normal((1, s.ngrad)) * 1e-6, dtype=torch.float32, device="cuda"))
            if len(rs) == 1:
                before = {mode: alone(0, mode) for mode in (1, 2)}
        for mode in (1, 2):
            want = [alone(i, mode) for i in range(2)]
            assert np.array_equal(want[0], before[mode])
            G = ReconGroup(rs)
            try:
                for R in rs:
                    R.reset()
                G.step_device([g.data_ptr() for g in gs])
                for a, b in zip(_commands(rs), want):
                    assert np.array_equal(a, b)
            finally:
                G.close()
    finally:
        for R in rs:
            R.close()
