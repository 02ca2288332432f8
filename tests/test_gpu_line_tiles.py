"""Line tiles at the edges of their parts: layers shared among the blocks of
a cluster, groups of spots and rounds that are not full, more layers than one
selection takes, LUT rows that are staged and rows that are not.

The dose does not depend on the split (bit for bit).  The 8x8x8 family keeps
its own code for all of this, so the line tiles are compared with it: the two
form the axis distance in different FP32 orders, 1e-5 of the maximum, as the
kernel shapes' own test has it."""
import copy
import ctypes

import numpy as np
import pytest
import torch

from conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DEV = torch.device("cuda", 0)


def _plan(n_layers, per_layer, depth_step=1.0, shape=(21, 37, 43), gantry=(30.0, 200.0)):
    """Beams of n_layers energies with per_layer spots each, water-like depths."""
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    model = copy.copy(IMPTPlan().beam_models[0])
    model.__dict__.pop("_pb_device_tables", None)
    model.lut_depths = (model.lut_depths * depth_step).astype(np.float32)
    if depth_step == 0.0:   # ascending, without a uniform step
        n = model.lut_depths.shape[1]
        model.lut_depths = np.tile((np.arange(n) + 0.3 * np.sin(np.arange(n))).astype(np.float32),
                                   (model.lut_depths.shape[0], 1))
    rng = np.random.default_rng(n_layers * 1000 + per_layer)
    rows = []
    for e in range(20, 20 + n_layers):
        xy = rng.uniform(-25.0, 25.0, (per_layer, 2))
        rows.append(np.column_stack([xy, rng.uniform(0.5, 1.5, per_layer),
                                     np.full(per_layer, e)]))
    spots = np.concatenate(rows).astype(np.float32)
    s = 3.0
    origin = -0.5 * s * np.array(shape[::-1], np.float32)
    dp = engine.DevicePlan(shape, s, origin,
                           [engine.BeamSpec(g, 0.0, np.zeros(3, np.float32), spots, model)
                            for g in gantry], DEV)
    j = torch.arange(shape[1], device=DEV, dtype=torch.float32)[None, :, None]
    i = torch.arange(shape[2], device=DEV, dtype=torch.float32)[None, None, :]
    wet = (0.3 * j + 0.01 * i + 1.0).expand(shape).reshape(1, -1).repeat(len(gantry), 1)
    dp.set_wet(wet.contiguous())
    return dp


def _dose(dp, split, order=True):
    from dosecuda_b200 import _lib
    out = torch.full((dp.n_vox,), float("nan"), device=DEV)
    _lib.check(_lib.lib.pb_dose_split(
        ctypes.byref(dp.grid), ctypes.cast(dp.beams, ctypes.c_void_p), dp.n_beams,
        _lib.ptr(dp.wet), _lib.ptr(dp.layers), _lib.ptr(dp.spot_geo), _lib.ptr(dp.mu_sorted), 1.0,
        _lib.ptr(out), _lib.ptr(dp.tile_order() if order else None), split,
        ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)))
    return out


@pytest.mark.parametrize("n_layers,per_layer,depth_step", [
    (1, 1, 1.0), (2, 5, 1.0), (3, 6, 1.0), (4, 7, 1.0), (5, 255, 1.0), (3, 256, 1.0),
    (2, 257, 1.0), (7, 13, 0.5), (3, 20, 0.7), (3, 20, 0.0), (33, 3, 1.0), (66, 2, 1.0)])
def test_splits_give_the_same_dose_and_match_the_other_family(n_layers, per_layer, depth_step):
    from dosecuda_b200 import _lib, autotune
    dp = _plan(n_layers, per_layer, depth_step)
    one = _dose(dp, 1)
    assert float(one.max()) > 0
    for split in (2, 4):
        assert torch.equal(_dose(dp, split), one)
        assert torch.equal(_dose(dp, split, order=False), one)
    other = dp.forward_variant(autotune.variants().index("t128_v4_c2"))
    assert torch.allclose(one, other, rtol=1e-5, atol=1e-5 * float(other.max()))

    w = torch.randn(dp.n_vox, device=DEV, generator=torch.Generator(DEV).manual_seed(3))
    ref = dp.adjoint(w, variant=autotune.variants().index("t128_v4_c2"))
    grad = torch.empty(dp.n_spots, device=DEV)
    for split in (1, 2, 4):
        _lib.check(_lib.lib.pb_dose_adjoint_split(
            ctypes.byref(dp.grid), ctypes.cast(dp.beams, ctypes.c_void_p), dp.n_beams,
            _lib.ptr(dp.wet), _lib.ptr(dp.layers), _lib.ptr(dp.spot_geo), _lib.ptr(w), 1.0,
            _lib.ptr(grad), _lib.ptr(dp.tile_order()), split,
            ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)))
        assert float((grad - ref).abs().max()) <= 1e-5 * float(ref.abs().max())


def test_nan_and_infinite_depths_as_the_other_family():
    """A NaN depth gives a NaN dose there, an infinite one none, and neither
    touches another voxel."""
    from dosecuda_b200 import autotune
    dp = _plan(3, 40)
    clean = _dose(dp, 1)
    dp.wet[:, 100] = float("nan")
    dp.wet[:, 5000] = float("inf")
    dp._order = None
    other = dp.forward_variant(autotune.variants().index("t128_v4_c2"))
    for split in (1, 4):
        d = _dose(dp, split)
        assert bool(torch.isnan(d[100])) == bool(torch.isnan(other[100]))
        assert float(d[5000]) == float(other[5000]) == 0.0
        keep = torch.ones(dp.n_vox, dtype=torch.bool, device=DEV)
        keep[[100, 5000]] = False
        assert torch.allclose(d[keep], clean[keep], rtol=1e-6, atol=1e-6 * float(clean.max()))
