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


def _reference_gradients(dp, w):
    """Weight and position gradients of sum w D in FP64 (sorted order), from
    the physics of the dose: torch.autograd on the spots' positions."""
    nx, ny, nz = dp.grid.nx, dp.grid.ny, dp.grid.nz
    geo = dp.spot_geo.cpu().double().reshape(-1, 8).numpy()
    mu = dp.mu_sorted.double()
    x = torch.tensor(geo[:, 0], device=DEV, requires_grad=True)
    y = torch.tensor(geo[:, 1], device=DEV, requires_grad=True)
    m = mu.clone().requires_grad_(True)
    k, j, i = torch.meshgrid(*(torch.arange(n, device=DEV, dtype=torch.float64)
                               for n in (nz, ny, nx)), indexing="ij")
    total = 0.0
    for b in range(dp.n_beams):
        B, G = dp.beams[b], dp.beams[b].geom
        model = dp._spec[b].model
        p = [a.reshape(-1) * float(dp.grid.spacing) - float(G.iso[q])
             for q, a in enumerate((i, j, k))]
        xt = p[0] * G.costa - p[2] * G.sinta
        hy = p[0] * G.sinta + p[2] * G.costa
        X, Y, Z = -(xt * G.cosga + p[1] * G.singa), hy, p[1] * G.cosga - xt * G.singa
        wet = dp.wet[b].double() * 10.0
        dist = torch.sqrt(X * X + Y * Y + (0.5 * (G.vsadx + G.vsady) - Z) ** 2)
        for L in dp.layers_np[dp.layer_offsets[b]:dp.layer_offsets[b + 1]]:
            e, first = int(L["energy_id"]), B.spot_start + int(L["spot_start"])
            sl = slice(first, first + int(L["n_spots"]))
            r80 = float(model.divergence_params[e, 1])
            ca, cb, cc = (float(v) for v in model.divergence_params[e, 2:5])
            lut = [torch.as_tensor(np.asarray(t[e], np.float64), device=DEV)
                   for t in (model.lut_depths, model.lut_sigmas, model.lut_idds)]
            lo = torch.searchsorted(lut[0], wet).clamp(1, len(lut[0]) - 1)
            f = ((wet - lut[0][lo - 1]) / (lut[0][lo] - lut[0][lo - 1])).clamp(0.0, 1.0)
            sig, idd = (t[lo - 1] + f * (t[lo] - t[lo - 1]) for t in lut[1:])
            d = dist - wet + 0.7 * r80
            st2 = (ca * d * d + cb * d + cc + sig) ** 2
            c = wet.clamp(min=0.1).clamp(max=r80 - 0.1)
            sh = 2.85 + 0.0014 * r80 * torch.log(c + 3.0) + 0.06 * c - 7.4e-5 * c * c - \
                0.22 * r80 / (c - r80 - 5.0) ** 2
            wh = 0.052 * torch.log(1.13 + c / (11.2 - 0.023 * r80)) + \
                0.35 * (0.0017 * r80 * r80 - r80) / ((r80 + 3.0) ** 2 - c * c) - \
                1.61e-9 * c * (r80 + 3.0) ** 2
            sh, wh = sh.clamp(min=0.0), wh.clamp(0.0, 0.9)
            sht2 = st2 + sh * sh
            tx, ty = x[sl] / G.vsadx, y[sl] / G.vsady
            ax = X[:, None] - x[sl] * (1.0 - Z / G.vsadx)[:, None]
            ay = Y[:, None] - y[sl] * (1.0 - Z / G.vsady)[:, None]
            az = tx * Y[:, None] - ty * X[:, None] - \
                x[sl] * y[sl] * (1.0 / G.vsadx - 1.0 / G.vsady)
            r2 = (ax * ax + ay * ay + az * az) / (1.0 + tx * tx + ty * ty)
            unit = idd / (2.0 * np.pi)
            kern = ((1.0 - wh) * unit / st2)[:, None] * torch.exp(-0.5 * r2 / st2[:, None]) + \
                (wh * unit / sht2)[:, None] * torch.exp(-0.5 * r2 / sht2[:, None])
            use = torch.where(wet <= float(np.float32(1.1) * np.float32(r80)), w.double(), 0.0)
            total = total + (use[:, None] * kern * m[sl]).sum()
    total.backward()
    return m.grad, x.grad, y.grad


@pytest.mark.parametrize("n_layers,per_layer,depth_step,shape", [
    (1, 1, 1.0, (21, 37, 43)), (2, 7, 1.0, (8, 16, 8)), (3, 9, 0.7, (9, 17, 9)),
    (2, 257, 1.0, (7, 15, 25)), (34, 5, 1.0, (12, 20, 17))])
def test_position_gradients_against_64_bits(n_layers, per_layer, depth_step, shape):
    """Every split, with and without an order, and without the weight
    gradient.  A gradient is a sum of some 1e4 to 1e5 signed FP32 terms, each
    with a few roundings and an exp2 of 2^-22: 1e-5 of the largest covers
    them (the terms' own magnitudes add up to some ten times the sum)."""
    from dosecuda_b200 import _lib
    dp = _plan(n_layers, per_layer, depth_step, shape)
    w = torch.randn(dp.n_vox, device=DEV, generator=torch.Generator(DEV).manual_seed(3)) + 0.5
    ref = _reference_gradients(dp, w)
    out = [torch.empty(dp.n_spots, device=DEV) for _ in range(3)]
    for split in (1, 2, 4):
        for order in (None, dp.tile_order()):
            weight = out[0] if order is None else None
            for o in out:
                o.fill_(float("nan"))
            _lib.check(_lib.lib.pb_dose_adjoint_positions_split(
                ctypes.byref(dp.grid), ctypes.cast(dp.beams, ctypes.c_void_p), dp.n_beams,
                _lib.ptr(dp.wet), _lib.ptr(dp.layers), _lib.ptr(dp.spot_geo),
                _lib.ptr(dp.mu_sorted), _lib.ptr(w), 1.0, _lib.ptr(weight), _lib.ptr(out[1]),
                _lib.ptr(out[2]), _lib.ptr(order), split,
                ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)))
            for q, (o, r) in enumerate(zip(out, ref)):
                if q > 0 or weight is not None:
                    assert float((o.double() - r).abs().max()) <= 1e-5 * float(r.abs().max())


@pytest.mark.parametrize("n_beams,n_layers", [(4, 1), (3, 2), (4, 3), (3, 4), (4, 5), (3, 33)])
def test_splits_with_uneven_layers_over_many_beams(n_beams, n_layers):
    """The cluster's blocks out of step: a layer of many compaction rounds
    beside layers that are left out (their spots lie outside the tiles' reach),
    staged beside unstaged LUT rows, an odd number of rounds in a beam and more
    layers than one selection takes.  Every launch gives the bits of split 1."""
    from dosecuda_b200 import engine
    from dosecuda_b200.plan_impt import IMPTPlan
    shape, s = (24, 40, 48), 3.0
    rng = np.random.default_rng(10 * n_beams + n_layers)
    beams = []
    for b in range(n_beams):
        model = copy.copy(IMPTPlan().beam_models[0])
        model.__dict__.pop("_pb_device_tables", None)
        if b % 2:   # rows that are not staged
            model.lut_depths = (model.lut_depths * 0.7).astype(np.float32)
        rows = []
        for q in range(n_layers):
            heavy = q == b % n_layers
            n = (1600 if n_layers < 9 else 600) if heavy else 3
            xy = rng.uniform(-20.0, 20.0, (n, 2))
            if not heavy and q % 2:
                # two corners of a box that the tiles lie in: selected, then left out
                xy = np.array([[-160.0, -160.0], [160.0, 160.0], [160.0, -160.0]])
            rows.append(np.column_stack([xy, rng.uniform(0.5, 1.5, n), np.full(n, 20.0 + q)]))
        beams.append(engine.BeamSpec(360.0 / n_beams * b + 7.0, 0.0, np.zeros(3, np.float32),
                                     np.concatenate(rows).astype(np.float32), model))
    dp = engine.DevicePlan(shape, s, -0.5 * s * np.array(shape[::-1], np.float32), beams, DEV)
    j = torch.arange(shape[1], device=DEV, dtype=torch.float32)[None, :, None]
    wet = (0.2 * j + 1.0).expand(shape).reshape(1, -1).repeat(n_beams, 1)
    dp.set_wet(wet.contiguous())
    one = _dose(dp, 1)
    assert float(one.max()) > 0
    for split in (2, 4):
        for rep in range(60):
            assert torch.equal(_dose(dp, split, order=rep % 2 == 0), one), (split, rep)


def _field(dp, kind):
    w = torch.randn(dp.n_vox, device=DEV, generator=torch.Generator(DEV).manual_seed(3)) + 0.5
    at = torch.arange(dp.n_vox, device=DEV)
    if kind == "none":
        w.zero_()
    elif kind == "one":
        w[at != dp.n_vox // 2] = 0.0
    elif kind == "part":
        w[at % (dp.grid.nx * dp.grid.ny) < dp.grid.nx * dp.grid.ny // 2] = 0.0
    return w


def _live_tiles(dp, w):
    g = dp.grid
    v = torch.nn.functional.pad((w.reshape(1, 1, g.nz, g.ny, g.nx) != 0).float(),
                                (0, -g.nx % 8, 0, -g.ny % 16, 0, -g.nz % 8))
    return int(torch.nn.functional.max_pool3d(v, (8, 16, 8)).sum())


@pytest.mark.parametrize("kind", ["none", "one", "part", "full"])
@pytest.mark.parametrize("n_layers,per_layer,shape", [(5, 20, (21, 37, 43)), (3, 300, (8, 16, 8)),
                                                      (7, 2, (9, 17, 9))])
def test_gradients_by_the_fields_tiles(kind, n_layers, per_layer, shape):
    """Every number of blocks that the count of the field's tiles can ask for, at
    the limits themselves, against one block per tile (atomic sums in another
    order: 1e-5 of the largest), with the count after a gradient's last entry
    and in a buffer of its own."""
    from dosecuda_b200 import _lib
    dp = _plan(n_layers, per_layer, shape=shape)
    w = _field(dp, kind)
    live = _live_tiles(dp, w)
    n = dp.n_spots
    stream = ctypes.c_void_p(torch.cuda.current_stream(DEV).cuda_stream)
    head = (ctypes.byref(dp.grid), ctypes.cast(dp.beams, ctypes.c_void_p), dp.n_beams,
            _lib.ptr(dp.wet), _lib.ptr(dp.layers), _lib.ptr(dp.spot_geo))
    order = _lib.ptr(dp.tile_order())
    ref = [torch.empty(n, device=DEV) for _ in range(3)]
    _lib.check(_lib.lib.pb_dose_adjoint_positions_split(
        *head, _lib.ptr(dp.mu_sorted), _lib.ptr(w), 1.0, *(_lib.ptr(r) for r in ref), order, 1,
        stream))
    assert (kind == "none") == (float(ref[0].abs().max()) == 0.0)

    def close(got):
        for a, b in zip(got, ref):
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())

    many = 1 << 20
    for limits in ((0, 0), (live, live), (live - 1, live), (live - 1, live - 1), (0, live),
                   (0, live - 1), (0, many), (live - 1, many), (many, many)):
        if limits[0] < 0 or limits[1] < limits[0]:
            continue
        lim = (ctypes.c_int * 2)(*limits)
        for apart in (False, True):
            out = [torch.full((n + 1,), float("nan"), device=DEV) for _ in range(3)]
            count = torch.full((1,), -5, dtype=torch.int32, device=DEV)
            at = count if apart else out[0][n:]
            _lib.check(_lib.lib.pb_dose_adjoint_field(
                *head, _lib.ptr(w), 1.0, _lib.ptr(out[0]), order, lim, _lib.ptr(at), stream))
            close([out[0][:n]])
            if apart and limits[0] == live - 1 and limits[1] == live and live > 1:
                assert int(count) == live
            at = count if apart else out[2][n:]
            for o in out:
                o.fill_(float("nan"))
            _lib.check(_lib.lib.pb_dose_adjoint_positions_field(
                *head, _lib.ptr(dp.mu_sorted), _lib.ptr(w), 1.0, *(_lib.ptr(o) for o in out),
                order, lim, _lib.ptr(at), stream))
            close([o[:n] for o in out])
    close([dp.adjoint(w)])
    close([dp.adjoint(w, out=torch.empty(n, device=DEV))])
    close(dp.adjoint_positions(w))
