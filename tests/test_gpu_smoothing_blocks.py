"""The smoothing's blocks at the edges of their parts: volumes without an
inside (every voxel in the shell), with one of a few voxels, with rows shorter
and longer than a warp's runs, several beams in one launch, and the batch.
Bit for bit the oracle's FP32-sum smoothing of the same raw depths."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DEV = torch.device("cuda", 0)


def _plan(shape, spacing, angles):
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    model = IMPTPlan().beam_models[0]
    iso = (0.5 * spacing * np.array(shape[::-1])).astype(np.float32)
    spots = np.array([[0.0, 0.0, 1.0, 30.0]], np.float32)
    dp = engine.DevicePlan(shape, spacing, np.zeros(3, np.float32),
                           [engine.BeamSpec(g, c, iso, spots, model) for g, c in angles], DEV)
    return dp, model, iso


def _rlsp(shape, seed):
    # depths on both sides of 1 cm, where the radii set in
    r = np.random.default_rng(seed).uniform(0.0, 0.6, shape).astype(np.float32)
    r[:, : shape[1] // 2] *= 4.0
    return torch.as_tensor(r, device=DEV).reshape(-1)


def _check(oracle, dp, model, iso, angles, shape, spacing):
    raw = dp.raw_wet.cpu().numpy().reshape(-1, *shape)
    got = dp.wet.cpu().numpy().reshape(-1, *shape)
    for b, (gantry, couch) in enumerate(angles):
        ob = oracle.beam_setup(gantry, couch, float(model.VSADX), float(model.VSADY), iso,
                               np.zeros(3, np.float32))
        want = oracle.smooth_f32(raw[b], spacing, ob)
        assert np.array_equal(got[b].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("shape,spacing", [
    ((5, 40, 33), 1.0), ((1, 1, 1), 2.0), ((23, 23, 23), 1.0), ((21, 22, 24), 1.0),
    ((12, 13, 300), 2.0), ((31, 17, 14), 2.0), ((9, 130, 12), 3.0), ((40, 8, 31), 4.0),
    ((14, 15, 16), 1.5)])
def test_shell_and_inside(oracle, shape, spacing):
    angles = [(0.0, 0.0), (270.0, 0.0), (31.0, 12.0)]
    dp, model, iso = _plan(shape, spacing, angles)
    dp.compute_wet(_rlsp(shape, 7), wet_mode="exact")
    _check(oracle, dp, model, iso, angles, shape, spacing)


def test_batch_of_uneven_volumes(oracle):
    from dosecuda_b200 import batch
    cases = [((5, 40, 33), 1.0, [(90.0, 0.0)]), ((31, 40, 27), 2.0, [(0.0, 0.0), (77.0, 5.0)]),
             ((3, 2, 1), 3.0, [(180.0, 0.0)]), ((24, 25, 26), 1.0, [(200.0, 340.0)])]
    plans, rlsps, more = [], [], []
    for q, (shape, spacing, angles) in enumerate(cases):
        dp, model, iso = _plan(shape, spacing, angles)
        rlsp = _rlsp(shape, q)
        dp.compute_wet(rlsp, wet_mode="texture" if q % 2 else "exact")
        alone = dp.wet.clone()
        plans.append(dp)
        rlsps.append(rlsp)
        more.append((model, iso, angles, shape, spacing, alone))
    batch.BatchPlans(plans, rlsps).run()
    torch.cuda.synchronize()
    for dp, (model, iso, angles, shape, spacing, alone) in zip(plans, more):
        _check(oracle, dp, model, iso, angles, shape, spacing)
        assert torch.equal(dp.wet, alone)


@pytest.mark.parametrize("shape,spacing", [((31, 57, 49), 1.0), ((70, 9, 141), 2.5),
                                           ((24, 240, 15), 2.0)])
def test_many_beams_as_each_alone(oracle, shape, spacing):
    """A launch large enough for four voxels a thread (16 beams) and ones that
    take two (a beam alone)."""
    angles = [(22.5 * b, 9.0 * (b % 4)) for b in range(16)]
    assert 16 * int(np.prod(shape)) > 2 * 148 * 9 * 512 / 1.1
    dp, model, iso = _plan(shape, spacing, angles)
    dp.compute_wet(_rlsp(shape, 3), wet_mode="exact")
    _check(oracle, dp, model, iso, angles, shape, spacing)
    for b in (0, 4, 11):
        one, _, _ = _plan(shape, spacing, angles[b:b + 1])
        one.compute_wet(_rlsp(shape, 3), wet_mode="exact")
        assert torch.equal(one.wet[0], dp.wet[b])


@pytest.mark.parametrize("n_plans", [5, 6, 7])
def test_batches_around_the_two_voxel_line(oracle, n_plans):
    """Batches of some 1.2 to 1.5 million voxels times beams, smoothed with two
    and with four voxels a thread: each plan's depths alone."""
    from dosecuda_b200 import batch
    angles = [(33.0, 0.0), (90.0, 5.0)]
    plans, rlsps, alone = [], [], []
    for q in range(n_plans):
        shape = (41 + q, 53, 47)
        dp, model, iso = _plan(shape, 2.0, angles)
        rlsp = _rlsp(shape, q)
        dp.compute_wet(rlsp, wet_mode="texture" if q % 2 else "exact")
        alone.append(dp.wet.clone())
        plans.append(dp)
        rlsps.append(rlsp)
        if q == 0:
            _check(oracle, dp, model, iso, angles, shape, 2.0)
    for dp in plans:
        dp.wet.fill_(float("nan"))
    batch.BatchPlans(plans, rlsps).run()
    torch.cuda.synchronize()
    for dp, wet in zip(plans, alone):
        assert torch.equal(dp.wet, wet)
