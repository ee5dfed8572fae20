"""The ghost-free periodic step on the GPU against the oracle, which copies
ghosts after every step: sizes below, at and past one 128-cell tile, boxes two
cells thin, call lengths that mix single steps, step pairs and the first step
of a state whose ghosts disagree, and every storage."""
import math

import numpy as np
import pytest
import torch

import lbm3_b200 as L
from lbm3_b200 import _abi as A
import oracle as O
from helpers import FIELD_REL_L2, density_velocity_errors, rel_l2

pytestmark = pytest.mark.gpu


def _case(dims, storage=A.LBM_STORE_F32):
    """A smooth wave whose ghosts hold the same values as their sources up to rounding."""
    c = L.periodic_box(*dims, nu_lattice=0.02, storage=storage)
    c.gx = 1e-6

    def initial(bc, i, j, k, info):
        a, b, d = (2 * math.pi * v / n for v, n in zip((i, j, k), dims))
        bc.dRho = 1e-3 * math.cos(a - b)
        bc.ux, bc.uy, bc.uz = 0.03 * math.sin(b + d), 0.02 * math.cos(a), 0.025 * math.sin(a - d)
    return L.set_hooks(c, initial_condition=initial)


@pytest.mark.parametrize("dims", [(2, 2, 2), (6, 10, 4), (8, 4, 4), (34, 6, 2), (30, 14, 18)])
def test_matches_oracle(dims):
    c = _case(dims)
    o = O.OracleGrid(c)
    with L.build_grids(c) as g:
        for steps in (1, 1, 2, 5):
            g.update_all_grids(steps)
            o.step(steps)
            e_rho, e_u, d_rho = density_velocity_errors(g.macro(), o.macro())
            assert e_rho < FIELD_REL_L2 and e_u < FIELD_REL_L2 and d_rho < 1e-6, (steps, e_rho, e_u, d_rho)
        # the ghosts repeat their sources after every call
        m = g.macro()
        np.testing.assert_array_equal(m[:, g.array("periodic_index")], m[:, g.array("periodic_source")])
        # a written state whose ghosts disagree steps with ghost copies first
        f = o.populations()
        f[:, 0] += np.float32(1e-4)
        o.set_populations(f)
        g.set_populations(f)
        g.update_all_grids(3)
        o.step(3)
        e_rho, e_u, _ = density_velocity_errors(g.macro(), o.macro())
        assert e_rho < FIELD_REL_L2 and e_u < FIELD_REL_L2, (e_rho, e_u)
    o.close()


@pytest.mark.parametrize("storage,tol", [(A.LBM_STORE_F64, 2e-6), (A.LBM_STORE_F16, 5e-3), (A.LBM_STORE_BF16, 4e-2)])
def test_storages_agree(storage, tol):
    """Against FP32 after 9 steps.  Rounding: FP32 keeps 2^-24 of a population
    per step, FP16 2^-11, BF16 2^-8; 9 steps of independent errors on
    velocities an order of magnitude below the populations' sum stay below
    ten units of it."""
    with L.build_grids(_case((30, 14, 18))) as a, L.build_grids(_case((30, 14, 18), storage)) as b:
        a.update_all_grids(9)
        b.update_all_grids(4)
        b.update_all_grids(5)
        assert rel_l2(b.macro()[1:4].reshape(-1), a.macro()[1:4].reshape(-1)) < tol


def test_batch_of_periodic_members():
    """More members than one launch holds, with a channel among them: each
    ends where it ends as a batch of its own, from states whose ghosts agree
    and states whose ghosts do not."""
    def cases():
        out = [_case((6 + 2 * (q % 4), 8, 4 + 2 * (q % 3)), A.LBM_STORE_F16) for q in range(17)]
        return out + [L.periodic_box(10, 8, 6, ux=0.03, storage=A.LBM_STORE_F16),
                      L.open_channel(16, 8, 8, storage=A.LBM_STORE_F16)]
    grids = [L.build_grids(c) for c in cases()]
    with L.PackedBatch(grids) as b:
        for steps in (1, 2, 3):
            b.update(steps)
    for c, g in zip(cases(), grids):
        with L.build_grids(c) as alone:
            with L.PackedBatch([alone]) as b:
                for steps in (1, 2, 3):
                    b.update(steps)
            np.testing.assert_array_equal(alone.populations(), g.populations())
        g.close()


@pytest.mark.parametrize("storage", [A.LBM_STORE_F32, A.LBM_STORE_F64])
def test_captured_steps_replay_on_written_state(storage):
    """Steps in a program's own graph, captured when the ghosts repeat their
    sources and replayed on populations whose ghosts do not.  Tolerance: a few
    single-precision roundings (6e-8 each) of shifted populations below 0.1; a
    step from the wrong ghosts is off by 1e-2 of them."""
    c = _case((8, 6, 4), storage)
    stream = torch.cuda.Stream()
    with L.build_grids(c) as g, L.build_grids(c) as ref:
        for x in (g, ref):
            x.update_all_grids(2)
            x.synchronize()
        g.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            g.update_all_grids(1)
            g.update_all_grids(1)
        f = g.populations()
        f *= 1 + 1e-2 * np.random.default_rng(5).standard_normal(f.shape).astype(np.float32)
        for x in (g, ref):
            x.set_populations(f)
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        ref.update_all_grids(4)
        np.testing.assert_allclose(g.macro(), ref.macro(), rtol=0, atol=2e-7)
        del graph


def test_batch_timed_over_no_steps():
    """A written state whose ghosts disagree, timed over no steps, then
    advanced: as the oracle advances it."""
    c = _case((8, 6, 4))
    o = O.OracleGrid(c)
    f = o.populations()
    f *= 1 + 1e-2 * np.random.default_rng(3).standard_normal(f.shape).astype(np.float32)
    o.set_populations(f)
    with L.build_grids(c) as g:
        g.set_populations(f)
        with L.PackedBatch([g]) as b:
            b.time_steps(0)
            b.update(3)
        o.step(3)
        e_rho, e_u, _ = density_velocity_errors(g.macro(), o.macro())
        assert e_rho < FIELD_REL_L2 and e_u < FIELD_REL_L2, (e_rho, e_u)
    o.close()


@pytest.mark.parametrize("storage", [A.LBM_STORE_F32, A.LBM_STORE_BF16])
def test_batch_with_one_written_member(storage):
    """Only the written member's ghosts differ: it steps with ghost copies, the
    others without, and each ends where it ends as a batch of its own."""
    cases = [_case((6 + 2 * q, 8, 4), storage) for q in range(3)]

    def run(grids, which):
        with L.PackedBatch(grids) as b:
            b.update(2)
            for q, g in zip(which, grids):
                if q == 1:
                    f = g.populations()
                    g.set_populations(f * (1 + 1e-2 * np.random.default_rng(6).standard_normal(f.shape).astype(np.float32)))
            for steps in (1, 1, 3):
                b.update(steps)
        return [g.populations() for g in grids]
    grids = [L.build_grids(c) for c in cases]
    together = run(grids, range(3))
    for q, c in enumerate(cases):
        with L.build_grids(c) as alone:
            np.testing.assert_array_equal(run([alone], [q])[0], together[q])
    for g in grids:
        g.close()
