"""Scenes at the edges of what the marches assume: opacities of every sign, maps whose
cells rounding makes empty, and the launch choices such scenes decide.

Bars: maps and sample counts equal the oracle's, every launch choice gives the same
image bit for bit (not-a-number included), and images stay within the exact form's bar
(max |dRGBA| <= 2e-3, >= 99.9% of pixels identical).
"""
import dataclasses

import numpy as np
import pytest

from oracle import mlp_oracle as M
from oracle.oracle import Oracle, render_bricks
from pilot_b200 import beams as B
from pilot_b200 import scenes
from test_marches_gpu import DTYPES, LIGHTS, frame, oracle, renderer, same, sparse
from test_rectilinear_gpu import check
from test_zz_no_alloc import _render_noalloc, _render_regular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nextra", [0, 2])
def test_opacities_that_are_never_positive(cuda_device, nextra):
    """No positive opacity: the maps are 0, but the view march composites the negative ones."""
    dims = (33, 20, 25)
    s = dataclasses.replace(scenes.small(41, n=24, image=48, m=9, kind="noise"), dims=dims, array=sparse(dims, 9))
    s.tf = s.tf.copy()
    s.tf[:, 3] = np.where(np.arange(len(s.tf)) < 90, 0.0, -0.1)
    with renderer(s) as r:
        for kind, v in LIGHTS[:nextra]:
            (r.add_directional_light if kind else r.add_point_light)(v, (0.3, 0.9, 0.5), 0.7)
        r.set_multi_light(nextra > 0)
        out = []
        for skip in (False, True):
            r.set_tuning(empty_skip=skip, view_skip=skip)
            img, t = r.render(s.camera())
            out.append((img, r.get_shadow_map((nextra + 1) * 1000), (t["light_samples"], t["lit_samples"])))
        assert np.min(out[0][0][..., 3]) < 0
        same(out[1], out[0], "leaps")
    if nextra == 0:
        oimg, lit = Oracle(s).view_march(Oracle(s).light_march()[0])
        assert out[1][2][1] == lit
        check(out[1][0], oimg)


def far(s, org, sp):
    """s with its field placed at org with the spacing sp."""
    at = lambda p: tuple(o + c * (n - 1) * sp for o, c, n in zip(org, p, s.dims))
    return dataclasses.replace(s, origin=org, brick_spacing=(sp,) * 3, cam_pos=at(s.cam_pos), cam_look=at(s.cam_look),
                               light=at(s.light) if s.light_kind == 0 else s.light,
                               sample_distance=s.sample_distance * (s.dims[0] - 1) * sp)


@pytest.mark.parametrize("lights", [1, 3])
@pytest.mark.parametrize("org", [(0.0, 0.0, 0.0), (4.0e3, 0.0, 9.0e3), (5.0e4, 0.0, 0.0)], ids=str)
def test_maps_finer_than_their_coordinates(cuda_device, org, lights):
    """Cells of 0.02 in a map 16 times as fine: near the coordinate origin every map cell has
    a width, 50,000 away most have none, and a sample in such a cell has no shading (not a
    number, whatever its opacity)."""
    s = far(dataclasses.replace(scenes.small(45, n=9, image=48, m=4, kind="blobs"), map_m=(128, 128, 128)), org, 0.02)
    with renderer(s) as r:
        for i in range(1, lights):
            r.add_directional_light(LIGHTS[i][1], (0.3, 0.9, 0.5), 0.7)
        r.set_multi_light(lights > 1)
        r.set_tuning(empty_skip=False, view_skip=False)
        img, t = r.render(s.camera())
        maps = r.get_shadow_map(lights * 129 ** 3)
        r.set_tuning(empty_skip=True, view_skip=True)
        again, t2 = r.render(s.camera())
        assert t2["lit_samples"] == t["lit_samples"]
        if lights > 1:
            assert np.array_equal(again, img, equal_nan=True)
    o = Oracle(s)
    if lights == 1:
        oimg, lit = o.view_march(maps.reshape(129, 129, 129))
    else:
        lc = np.stack([np.float32(s.light_color) * np.float32(s.light_intensity)]
                      + [np.float32((0.3, 0.9, 0.5)) * np.float32(0.7)] * (lights - 1))
        oimg, lit = o.view_march_multi(maps.reshape(lights, -1), lc)
    assert t["lit_samples"] == lit and np.isnan(oimg).any() == (org[0] > 1e4)
    nan = np.isnan(oimg)
    assert np.mean(np.isnan(img) == nan) > 0.999
    check(np.where(nan, 0, img), np.where(nan, 0, oimg))


@pytest.mark.parametrize("log2", [10, 13])
def test_batches_larger_than_the_training_set(cuda_device, log2):
    """A step takes at most the whole set: 15/16 of the samples, the rest is held out. Bar: as
    a batch of just that size, whatever an earlier, larger training left behind (the sums'
    order varies, which four steps of 1e-3 keep below 1% of the error)."""
    s = scenes.small(46, n=24, image=16, m=8)
    size = (1 << log2) - (1 << (log2 - 4))
    with renderer(s) as r:
        r.mlp_train(B.mlp_options(samples_log2=16, epochs=1, batch=16384, lr=1e-3))
        reps = [r.mlp_train(B.mlp_options(samples_log2=log2, epochs=4, batch=b, lr=1e-3)) for b in (size, size + 1, 1 << 20)]
    for rep in reps:
        assert rep["steps"] == 4 and rep["initial_rmse"] == pytest.approx(reps[0]["initial_rmse"], rel=1e-5)
        assert abs(rep["holdout_rmse"] - reps[0]["holdout_rmse"]) <= 0.01 * reps[0]["holdout_rmse"]


def test_training_set_given_back_when_memory_runs_out(cuda_device):
    """The set kept for the next training goes when a buffer of the renderer cannot be had; with
    nothing kept the call fails as before, and the next training allocates its set again."""
    s = scenes.small(47, n=24, image=16, m=8)
    opts = B.mlp_options(samples_log2=12, epochs=1, batch=1024, lr=1e-3)
    with renderer(s) as r:
        r.render(s.camera())
        r.mlp_train(opts)
        for m in (20, 30):
            r.set_shadow_map_size(m)  # a larger map buffer
            B.lib().beams_test_fail_allocation(1)
            try:
                if m == 20:
                    r.render(s.camera())
                else:
                    with pytest.raises(B.BeamsError, match="OOM"):
                        r.render(s.camera())
            finally:
                B.lib().beams_test_fail_allocation(0)
        img, _ = r.render(s.camera())
        assert r.mlp_train(opts)["steps"] == 3
        again, _ = r.render(s.camera())
    assert np.array_equal(img, again)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_hidden_units_that_are_not_numbers_are_off(cuda_device, value):
    """The march's network clamps a sum that is not a number to 0. Bar: the image of the network
    whose units are switched off by their biases, bit for bit."""
    s = scenes.small(49, n=24, image=24, m=8)
    P = np.random.default_rng(49).normal(0, 0.08, M.N_PARAMS).astype(np.float32)

    off, odd = P.copy(), P.copy()
    for layer, unit in (("1", 3), ("2", 9), ("3", 17), ("4", 40)):
        w, b = M.OFF["W" + layer][0], M.OFF["B" + layer][0]
        off[b + unit] = -1e30
        # weights of the value and of its opposite (two infinities that meet sum to NaN), and the bias
        odd[w + unit], odd[w + 64 + unit], odd[b + unit] = value, -value, np.nan
    out = []
    with renderer(s) as r:
        for p in (off, odd):
            r.mlp_set_params(p)
            r.set_form(B.FORM_MLP, B.mlp_options(knot=1, probe_fraction=0.0))
            out.append(r.render(s.camera())[0])
    assert np.isfinite(out[0]).all() and np.array_equal(out[1], out[0])


@pytest.mark.parametrize("ny", [745, 748])
def test_learned_form_on_the_longest_axes(cuda_device, ny):
    """A knot of 64 fits beside 9,963 table entries (cells and colours), the axes' closing ones not
    counted. Bar: on rays of fewer lit samples than the knot, the image of a knot of 63 (which
    leaves room to spare), bit for bit."""
    dims = (8192, ny, 2)
    s = dataclasses.replace(scenes.small(53, n=24, image=40, m=8, kind="noise"), dims=dims, sample_distance=0.03,
                            array=np.random.default_rng(53).random(dims[::-1], np.float32))
    s.tf = np.repeat(s.tf, -(-1024 // len(s.tf)), axis=0)[:1024]
    assert len(s.tf) + sum(dims) - 3 in (9960, 9963)
    P = np.random.default_rng(53).normal(0, 0.08, M.N_PARAMS).astype(np.float32)
    out = []
    with renderer(s) as r:
        r.mlp_set_params(P)
        for knot in (63, 64):
            r.set_form(B.FORM_MLP, B.mlp_options(knot=knot, probe_fraction=0.0))
            out.append(r.render(s.camera()))
    assert np.max(out[0][0][..., 3]) > 0 and out[0][1]["lit_samples"] == out[1][1]["lit_samples"]
    assert np.array_equal(out[1][0], out[0][0])


@pytest.mark.parametrize("name,dt", DTYPES[:2], ids=lambda d: str(d))
@pytest.mark.parametrize("org", [(3.0e5, 0.0, 1.0e3), (4.0e6, 2.5e6, 0.0), (0.0, 3.0e7, 5.0e6)], ids=str)
def test_positions_rounded_onto_faces(cuda_device, org, name, dt):
    """Cells of width 1 far from the coordinate origin: positions are multiples of 1/32, of 1/4
    and 1/2, and of 2 (where cells have width 0 or 2), so samples lie on faces and edges."""
    s = far(dataclasses.replace(scenes.small(50, n=21, image=40, m=8, kind="noise"), map_m=(9, 11, 8)), org, 1.0)
    o = oracle(s, name)
    om, _ = o.light_march()
    oimg, lit = o.view_march(om)
    with renderer(s, dt) as r:
        for skip in (False, True):
            r.set_tuning(empty_skip=skip, view_skip=skip)
            img, m, n = frame(r, s)
            assert np.array_equal(m, om.ravel()) and n[1] == lit, skip
            nan = np.isnan(oimg)
            assert np.array_equal(np.isnan(img), nan)
            check(np.where(nan, 0, img), np.where(nan, 0, oimg))


@pytest.mark.parametrize("light", [(0, (0.5, 0.5, 0.5)), (0, (0.0, 0.5, 1.0)), (0, (1.0, 0.25, 0.5)), (0, (2.0, 0.5, 0.5)),
                                   (0, (1e25, 0.0, 0.0)), (1, (0.3, -0.8, 0.1))], ids=str)
def test_bricks_lit_from_one_of_their_vertices(cuda_device, light):
    """The ray to a vertex at the light has no direction and its stitched value is not a number, as
    are the shadings that read it, whatever the samples' opacity."""
    s = dataclasses.replace(scenes.small(51, n=33, image=40, m=8, kind="blobs"), light_kind=light[0], light=light[1])
    bricks = scenes.split_bricks(s, (2, 2, 2))
    oimg, _, _, maps, lit = render_bricks(bricks)
    with B.Renderer(0) as r:
        bricks[0].configure(r)
        r.set_bricks([(b.field_numpy(), b.origin, b.spacing, b.value_range) for b in bricks])
        img, t = r.render(s.camera())
        assert t["lit_samples"] == lit
        for b in range(len(bricks)):
            assert np.array_equal(r.get_brick_map(b, 1, 729), np.ravel(maps[b]), equal_nan=True), b
    nan = np.isnan(oimg)
    assert np.array_equal(np.isnan(img), nan)
    check(np.where(nan, 0, img), np.where(nan, 0, oimg))


@pytest.mark.parametrize("kind", ["jitter", "power", "wide"])
@pytest.mark.parametrize("dims", [(2, 3, 60), (41, 5, 2), (70, 33, 9)], ids=str)
@pytest.mark.parametrize("steps", [3.0, 40.0, 400.0])
def test_coordinate_searches_over_short_and_long_steps(cuda_device, kind, dims, steps):
    """From a fraction of a cell a step to most of the axis, up and down, on axes of a few cells."""
    rng = np.random.default_rng(sum(dims))
    t = [np.linspace(0.0, 1.0, n) for n in dims]
    coords = {"jitter": [np.concatenate([[0.0], (q[1:-1] + rng.uniform(-0.3, 0.3, len(q) - 2) / len(q)), [1.0]]) for q in t],
              "power": [q ** 4 for q in t],
              "wide": [np.concatenate([q[:-1] * 1e-2, [1.0]]) for q in t]}[kind]
    for light in ((0, (2.0, -1.0, 3.0)), (1, (1.0, 0.7, -0.6))):
        s = dataclasses.replace(scenes.small(52, n=9, image=40, m=7, kind="noise"), dims=dims, light_steps=steps,
                                array=rng.uniform(0, 1, dims[::-1]).astype(np.float32), sample_distance=2.0 / steps,
                                light_kind=light[0], light=light[1])
        s.coords = tuple(np.float32(c) for c in coords)
        for name, dt in DTYPES[:2]:
            o = oracle(s, name)
            om, _ = o.light_march()
            oimg, lit = o.view_march(om)
            with renderer(s, dt) as r:
                img, m, n = frame(r, s)
                assert np.array_equal(m, om.ravel()) and n[1] == lit, (light, name)
                check(img, oimg)
        cells = s.array[:-1, :-1, :-1].copy()
        oimg, lit = Oracle(s, field=cells).view_march_cells()
        with B.Renderer(0) as r:
            r.set_volume(cells, dims=dims, origin=s.origin, spacing=s.spacing, value_range=s.value_range, assoc=B.ASSOC_CELLS)
            r.set_volume_coordinates(*s.coords)
            s.configure(r)
            r.set_use_shadow_map(False)
            img, t = r.render(s.camera())
            assert t["lit_samples"] == lit
            check(img, oimg)


# split rays below 160,000 vertices; else columns where twice the vertices are the field's points
@pytest.mark.parametrize("dims,m", [((80, 80, 80), 53), ((80, 80, 80), 54), ((53, 71, 97), 55), ((41, 90, 95), 55),
                                    ((42, 90, 95), 55), ((9, 300, 70), 56), ((90, 90, 90), 70)], ids=str)
def test_allocation_free_frames_in_each_vertex_order(cuda_device, dims, m):
    """Bar: the regular entry point's image, bit for bit."""
    import torch
    rng = np.random.default_rng(sum(dims))
    for light in ((2.0, 0.4, 0.5), (0.3, -2.0, 0.9), (0.45, 0.5, 0.4)):
        s = dataclasses.replace(scenes.small(54, n=9, image=40, m=m, kind="noise"), dims=dims, light_kind=0, light=light,
                                array=rng.uniform(0, 1, dims[::-1]).astype(np.float32))
        fd, tf = torch.from_numpy(s.array).cuda(), torch.from_numpy(np.ascontiguousarray(s.tf, np.float32)).cuda()
        out = torch.full((s.height, s.width, 4), -1.0, device="cuda")
        assert _render_noalloc(s, fd, tf, out) == 0
        assert np.array_equal(out.cpu().numpy(), _render_regular(s))
