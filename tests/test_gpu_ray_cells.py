"""The ray trace's samples from the cell records.

With the texture unit's filter: compared with the unit itself over random
coordinates, over every pair of fractions of two axes, and at the halves of the
coordinates' 1/256 steps and of the weights, with volumes of one texel (each
weight by itself) and of noise.  Both sum at most eight products of a weight
(whole 256ths) and a texel in FP32: 8 roundings of the largest texel.

With exact weights: the depths of a noisy volume with and without the
records, whose samples are the same FP32 operations (sums of 4 and of 8 samples
before FP64: 1e-6 of the largest depth)."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

DEV = torch.device("cuda", 0)


def _samples(vol, at):
    """(unit, cells) of the volume (nz, ny, nx) at the coordinates (n, 3)."""
    from dosecuda_b200 import _lib
    nz, ny, nx = vol.shape
    g = _lib.PbGrid(nx, ny, nz, 1.0)
    h = ctypes.c_uint64(0)
    stream = ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)
    v = torch.as_tensor(vol, device=DEV).contiguous()
    _lib.check(_lib.lib.pb_texture_create(_lib.ptr(v), ctypes.byref(g), ctypes.byref(h), stream))
    try:
        a = torch.as_tensor(at, dtype=torch.float32, device=DEV).contiguous()
        assert len(a) % 2 == 0
        unit, cells = torch.empty(len(a), device=DEV), torch.empty(len(a), device=DEV)
        _lib.check(_lib.lib.pb_texture_sample(h, ctypes.byref(g), _lib.ptr(a), len(a) // 2,
                                              _lib.ptr(unit), _lib.ptr(cells), stream))
        torch.cuda.synchronize()
    finally:
        _lib.lib.pb_texture_destroy(h)
    return unit.cpu().numpy(), cells.cpu().numpy()


BOUND = 8.0 * 2.0 ** -24


@pytest.mark.parametrize("shape", [(24, 31, 40), (1, 5, 7), (3, 2, 1)])
def test_filter_is_the_units(shape):
    rng = np.random.default_rng(5)
    vol = rng.uniform(0.0, 2.0, shape).astype(np.float32)
    n = np.array(shape[::-1], np.float64)
    at = rng.uniform(0.0, 1.0, (1 << 18, 3)) * n
    at[::3] = np.floor(at[::3] * 1024.0) / 1024.0   # among them the halves of 1/256
    unit, cells = _samples(vol, at.astype(np.float32))
    assert unit.max() > 0.5
    assert np.abs(unit - cells).max() <= BOUND * vol.max()


def test_weights_of_every_texel():
    """One texel of 1: the sample is that texel's weight, a whole 256th."""
    vol = np.zeros((8, 8, 8), np.float32)
    vol[4, 4, 4] = 1.0
    f = np.arange(256) / 256.0
    rng = np.random.default_rng(2)
    for axes in ((0, 1), (0, 2), (1, 2)):
        for corner in range(8):
            at = np.empty((256 * 256, 3))
            for a in range(3):
                part = rng.integers(0, 256) / 256.0
                if a == axes[0]:
                    part = np.repeat(f, 256)
                elif a == axes[1]:
                    part = np.tile(f, 256)
                at[:, a] = 4.0 - ((corner >> a) & 1) + 0.5 + part
            unit, cells = _samples(vol, at)
            assert np.array_equal(unit, cells)
            assert np.array_equal(unit * 256.0, np.round(unit * 256.0))


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_not_a_number_and_infinite_texels(value):
    """The unit leaves out texels of weight 0, so a volume with such a value is
    sampled by the unit: the depths are those of the handle whose other texels
    are finite, wherever the ray does not come near it, and no ray that passes
    it loses a sample that the unit has."""
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    shape = (14, 16, 18)
    rng = np.random.default_rng(8)
    vol = rng.uniform(0.5, 1.5, shape).astype(np.float32)
    spots = np.array([[0.0, 0.0, 1.0, 30.0]], np.float32)
    iso = np.array([18.0, 16.0, 14.0], np.float32)
    dp = engine.DevicePlan(shape, 2.0, np.zeros(3, np.float32),
                           [engine.BeamSpec(0.0, 0.0, iso, spots, IMPTPlan().beam_models[0])], DEV)

    def raw(v):
        dp.compute_wet(torch.as_tensor(v, device=DEV).reshape(-1))
        return dp.raw_wet.clone().reshape(shape)
    clean = raw(vol)
    vol[7, 8, 9] = value
    other = raw(vol)
    far = torch.ones(shape, dtype=torch.bool, device=DEV)
    far[5:10, :, 7:12] = False
    assert torch.allclose(other[far], clean[far], rtol=2e-6, atol=1e-6)
    assert not torch.equal(torch.nan_to_num(other), torch.nan_to_num(clean))
    vol[7, 8, 9] = 1.0
    raw(vol)
    assert bool(torch.isfinite(dp.raw_wet).all())


@pytest.mark.parametrize("shape,spacing,angle,couch", [
    ((24, 30, 37), 2.5, 31.0, 12.0), ((19, 40, 33), 1.0, 0.0, 0.0), ((40, 9, 64), 3.0, 270.0, 0.0)])
@pytest.mark.parametrize("noise", [0.0, 0.02])
def test_exact_depths_with_and_without_records(shape, spacing, angle, couch, noise):
    from dosecuda_b200 import _lib, engine
    from dosecuda_b200.plan_impt import IMPTPlan
    rng = np.random.default_rng(3)
    rho = np.ones(shape, np.float32)
    rho[:, : shape[1] // 3] = 0.25
    rho += (noise * rng.standard_normal(shape)).astype(np.float32)
    iso = 0.47 * spacing * np.array(shape[::-1], np.float32)
    spots = np.array([[0.0, 0.0, 1.0, 30.0]], np.float32)
    dp = engine.DevicePlan(shape, spacing, np.zeros(3, np.float32),
                           [engine.BeamSpec(angle, couch, iso, spots, IMPTPlan().beam_models[0])],
                           DEV)
    v = torch.as_tensor(rho, device=DEV).reshape(-1).contiguous()
    dp.compute_wet(v, wet_mode="exact")
    with_records = dp.raw_wet.clone()
    raw, wet = torch.empty_like(with_records), torch.empty_like(with_records)
    _lib.check(_lib.lib.pb_wet(_lib.ptr(v), 0, ctypes.byref(dp.grid),
                               ctypes.cast(dp.geoms, ctypes.c_void_p), 1, _lib.ptr(raw),
                               _lib.ptr(wet), None,
                               ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)))
    assert float(raw.max()) > 1.0
    assert float((raw - with_records).abs().max()) <= 1e-6 * float(raw.max())


def _half_noisy(shape, planes, seed=4):
    """A volume with noise in its first `planes` planes and 1 in the others."""
    rng = np.random.default_rng(seed)
    vol = np.ones(shape, np.float32)
    vol[:planes] = rng.uniform(0.5, 1.5, (planes,) + shape[1:]).astype(np.float32)
    return vol


def _texture_plan(shape, spacing, angle):
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    iso = 0.47 * spacing * np.array(shape[::-1], np.float32)
    spots = np.array([[0.0, 0.0, 1.0, 30.0]], np.float32)
    return engine.DevicePlan(shape, spacing, np.zeros(3, np.float32),
                             [engine.BeamSpec(angle, 0.0, iso, spots, IMPTPlan().beam_models[0])],
                             DEV)


def _raw(dp, vol):
    dp.compute_wet(torch.as_tensor(vol, device=DEV).reshape(-1))
    return dp.raw_wet.clone().reshape(vol.shape)


@pytest.mark.parametrize("shape", [(40, 30, 33), (60, 17, 24), (160, 90, 70)])
@pytest.mark.parametrize("angle,spacing", [(0.0, 2.5), (90.0, 1.0), (37.0, 3.0)])
def test_sparse_and_dense_volumes_agree(shape, angle, spacing):
    """On either side of the share of cells that are not flat from which the
    samples come from the records too: two volumes that differ in their last
    planes alone give the same depths in the first ones, whose rays stay there
    (the couch is at 0, so rays run in z only by the divergence).  Samples agree
    to 8 roundings of the largest texel, their FP32 sums of 4 to 4 more: 1e-6 of
    the largest depth."""
    nz = shape[0]
    near = int(0.8 * nz)
    sparse, dense = _half_noisy(shape, near), _half_noisy(shape, nz)
    assert np.array_equal(sparse[:near], dense[:near])
    rough = (near + 2) / (nz + 1)           # cells of the noisy planes and their faces
    assert rough < 0.85
    dp = _texture_plan(shape, spacing, angle)
    a, b = _raw(dp, sparse), _raw(dp, dense)
    first = slice(0, near // 2)
    assert float(a[first].max()) > 1.0
    assert float((a[first] - b[first]).abs().max()) <= 1e-6 * float(b.max())
    assert not torch.equal(a[near + 2:], b[near + 2:])


def test_refilling_a_handle_with_the_other_kind():
    """One handle filled with a dense, a sparse, a flat and a dense volume
    again: the bits of handles of their own."""
    shape = (40, 31, 37)
    vols = [_half_noisy(shape, 40), _half_noisy(shape, 9), np.ones(shape, np.float32),
            _half_noisy(shape, 40, seed=9), _half_noisy(shape, 12)]
    dp = _texture_plan(shape, 2.0, 21.0)
    for vol in vols:
        got = _raw(dp, vol)
        assert torch.equal(got, _raw(_texture_plan(shape, 2.0, 21.0), vol))


@pytest.mark.parametrize("planes", [0, 30, 128])
@pytest.mark.parametrize("mode", ["texture", "exact"])
def test_many_bricks_give_each_beams_depths(planes, mode):
    """A launch with more bricks than get a block each (16 beams), one with a
    block each (a beam alone), sparse and dense: the same bits."""
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    shape = (121, 126, 123)
    vol = torch.as_tensor(_half_noisy(shape, min(planes, shape[0])), device=DEV).reshape(-1)
    iso = np.array(shape[::-1], np.float32)
    spots = np.array([[0.0, 0.0, 1.0, 30.0]], np.float32)
    model = IMPTPlan().beam_models[0]
    beams = [engine.BeamSpec(22.5 * b, 7.0 * (b % 3), iso, spots, model) for b in range(16)]
    dp = engine.DevicePlan(shape, 2.0, np.zeros(3, np.float32), beams, DEV)
    wet = dp.compute_wet(vol, wet_mode=mode)
    for b in (0, 5, 15):
        one = engine.DevicePlan(shape, 2.0, np.zeros(3, np.float32), [beams[b]], DEV)
        assert torch.equal(one.compute_wet(vol, wet_mode=mode)[0], wet[b])


@pytest.mark.parametrize("left", [25.7, 13.0, 2.0])
def test_grids_that_leave_little_memory(left):
    """A handle made where only `left` bytes a voxel are free beside its texture:
    with the records, or without any (pb_texture_create has to succeed), the
    depths of a handle with records.  Runs of samples and samples one by one
    add up in FP32 groups of 8 at most: 1e-6 of the largest depth."""
    shape = (300, 320, 320)
    v = int(np.prod(shape))
    vol = np.ones(shape, np.float32)
    vol[:, 100:180, 60:200] = 1.5
    dp = _texture_plan(shape, 2.0, 0.0)
    ref = _raw(dp, vol)
    rlsp = torch.as_tensor(vol, device=DEV).reshape(-1)
    del dp
    dp = _texture_plan(shape, 2.0, 0.0)
    torch.cuda.synchronize()
    # the depths' buffers come from torch's cache, the handle from what is left
    free = torch.cuda.mem_get_info(DEV)[0]
    hog = torch.empty(int(free - (4.3 + left) * v), dtype=torch.uint8, device=DEV)
    try:
        dp.compute_wet(rlsp)
        torch.cuda.synchronize()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert float((dp.raw_wet.reshape(shape) - ref).abs().max()) <= 1e-6 * float(ref.max())


@pytest.mark.parametrize("noise", [0.0, 0.02])
def test_axis_past_the_filters_fixed_point(noise):
    """More than 8191 voxels along an axis: exact depths with and without records
    as above; texture depths within the unit's weights of them, which are off
    by 1/512 at most on each axis."""
    from dosecuda_b200 import _lib
    shape = (6, 7, 8200)
    rng = np.random.default_rng(3)
    rho = np.ones(shape, np.float32)
    rho[:, :, 3000:5000] = 0.25
    rho += (noise * rng.standard_normal(shape)).astype(np.float32)
    dp = _texture_plan(shape, 2.0, 0.0)
    v = torch.as_tensor(rho, device=DEV).reshape(-1).contiguous()
    dp.compute_wet(v)
    tex = dp.raw_wet.clone()
    at, out = torch.zeros(6, device=DEV), torch.zeros(2, device=DEV)
    stream = ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)
    assert _lib.lib.pb_texture_sample(dp._tex, ctypes.byref(dp.grid), _lib.ptr(at), 1,
                                      _lib.ptr(out), _lib.ptr(out), stream) == _lib.PB_ERR_INVALID
    dp.compute_wet(v, wet_mode="exact")
    exact = dp.raw_wet.clone()
    raw, wet = torch.empty_like(exact), torch.empty_like(exact)
    _lib.check(_lib.lib.pb_wet(_lib.ptr(v), 0, ctypes.byref(dp.grid),
                               ctypes.cast(dp.geoms, ctypes.c_void_p), 1, _lib.ptr(raw),
                               _lib.ptr(wet), None, stream))
    top = float(raw.max())
    assert top > 0.5
    assert float((raw - exact).abs().max()) <= 1e-6 * top
    assert float((tex - exact).abs().max()) <= 3.0 / 512.0 * float(rho.max()) / 0.2 * top


@pytest.mark.parametrize("shape", [(40, 30, 33), (160, 90, 70)])
@pytest.mark.parametrize("angle,spacing", [(0.0, 2.5), (37.0, 3.0)])
def test_sparse_and_dense_depths_are_the_same_bits(shape, angle, spacing):
    """As test_sparse_and_dense_volumes_agree: every sample is the unit's and the
    sums go the same way, so the depths are the same bits, smoothed ones too (a
    depth off by a rounding can decide a radius of the smoothing otherwise)."""
    nz = shape[0]
    near = int(0.8 * nz)
    dp = _texture_plan(shape, spacing, angle)
    first = slice(0, near // 2)
    out = []
    for planes in (near, nz):
        raw = _raw(dp, _half_noisy(shape, planes))
        out.append((raw[first], dp.wet.clone().reshape(shape)[first]))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1][:near // 2 - 12], out[1][1][:near // 2 - 12])
