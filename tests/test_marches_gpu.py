"""The marches where their launches and layouts change form: vertex orders and the
four-lanes-a-ray split around its thresholds, leaps over empty macro-cells, the
field copy at every tile remainder, samples that lie on cell faces, the reciprocal
division far from unit scale, coordinate searches from both starting points, and
the network's kernels around their tile sizes.

Bars: maps and sample counts equal the oracle's, and every launch choice gives the
same map, image and counts, bit for bit (the device executes the oracle's float32
operations in its order). Images against the oracle: the exact form's bar (max
|dRGBA| <= 2e-3, >= 99.9% of pixels identical, the ray set-up's float64 slab may
differ in the last place).
"""
import dataclasses

import numpy as np
import pytest

from oracle import mlp_oracle as M
from oracle.oracle import Oracle, quantize, render_bricks
from pilot_b200 import beams as B
from pilot_b200 import scenes
from test_rectilinear_gpu import check, stretched

pytestmark = pytest.mark.gpu
DTYPES = [("f32", None), ("bf16", B.BF16), ("f16", B.F16)]


def renderer(s, dt=None):
    r = B.Renderer(0)
    r.set_volume(s.field_numpy(), origin=s.origin, spacing=s.spacing, value_range=s.value_range)
    if getattr(s, "coords", None) is not None:
        r.set_volume_coordinates(*s.coords)
    s.configure(r)
    if dt is not None:
        r.set_form(B.FORM_PRECISION, field_dtype=dt)
    return r


def oracle(s, name):
    return Oracle(s) if name == "f32" else Oracle(s, field=quantize(s.field_numpy(), name), precision=True)


def frame(r, s):
    img, t = r.render(s.camera())
    m = s.map_m if isinstance(s.map_m, tuple) else (s.map_m,) * 3
    return img, r.get_shadow_map((m[0] + 1) * (m[1] + 1) * (m[2] + 1)), (t["light_samples"], t["lit_samples"])


def same(a, b, what):
    for x, y in zip(a[:2], b[:2]):
        assert np.array_equal(x, y, equal_nan=True), what
    assert a[2] == b[2], (what, a[2], b[2])


# the light along each axis and sign, oblique, and a point light inside the volume
LIGHTS = [(1, (0.05, -1.0, 0.02)), (1, (1.0, 0.0, 0.0)), (1, (-0.6, 0.59, -0.61)), (0, (0.4, 0.45, 0.6)),
          (0, (0.5, 0.5, 3.0))]


@pytest.mark.parametrize("m", [(1, 1, 1), (11, 7, 14), (2, 33, 8), (8, 8, 9)])
@pytest.mark.parametrize("light", LIGHTS, ids=str)
def test_every_vertex_order_builds_the_oracles_map(cuda_device, m, light):
    s = dataclasses.replace(scenes.small(31, n=20, image=16, m=4, kind="noise"), dims=(21, 18, 26), map_m=m,
                            light_kind=light[0], light=light[1], array=None)
    om, _ = Oracle(s).light_march()
    with renderer(s) as r:
        for brick in (0, 8, 16, 32, 64):
            for skip in (False, True):
                r.set_tuning(light_brick=brick, empty_skip=skip)
                r.render(s.camera())
                got = r.get_shadow_map(om.size)
                assert np.array_equal(got, om.ravel()), (brick, skip)


# The rays are split below 160,000 slots (exact) and 100,000 (precision). Slots of
# the 8-wide order: 51 56 56 and 52 56 56, 43 48 48 and 44 48 48; in rows: 54^3 and 55^3,
# 46^3 and 47^3.
@pytest.mark.parametrize("name,dt,m", [("f32", None, 50), ("f32", None, 51), ("f32", None, 53), ("f32", None, 54),
                                       ("bf16", B.BF16, 42), ("bf16", B.BF16, 43), ("f16", B.F16, 45),
                                       ("f16", B.F16, 46)])
def test_split_rays_around_the_thresholds(cuda_device, name, dt, m):
    s = scenes.small(32, n=28, image=32, m=m, kind="blobs")
    om, _ = oracle(s, name).light_march()
    with renderer(s, dt) as r:
        counts = set()
        for brick in (0, 8):
            for skip in (False, True):
                r.set_tuning(light_brick=brick, empty_skip=skip)
                _, t = r.render(s.camera())
                assert np.array_equal(r.get_shadow_map(om.size), om.ravel()), (brick, skip)
                counts.add(t["light_samples"])
        assert len(counts) == 1


@pytest.mark.parametrize("fov", [2.0, 20.0, 60.0])
def test_lists_of_vertices_short_and_long(cuda_device, fov):
    """A lazy map's list decides by its own length: from a few vertices to most of 73^3."""
    s = dataclasses.replace(scenes.small(33, n=32, image=64, m=72, kind="noise"), fov_y_deg=fov)
    with renderer(s) as r:
        for dt in (None, B.BF16):
            if dt is not None:
                r.set_form(B.FORM_PRECISION, field_dtype=dt)
            full, tf = r.render(s.camera())
            r.set_lazy_shadow_map(True)
            lazy, tl = r.render(s.camera())
            r.set_lazy_shadow_map(False)
            assert np.array_equal(full, lazy) and tl["lit_samples"] == tf["lit_samples"]
            print(f"fov {fov}: {tl['map_vertices']} of {73 ** 3} vertices")


def sparse(dims, seed):
    """Mostly empty: a few small bright boxes, some touching the last cells."""
    rng = np.random.default_rng(seed)
    f = np.zeros(dims[::-1], np.float32)
    for _ in range(5):
        lo = [int(rng.integers(0, n - 1)) for n in dims[::-1]]
        f[tuple(slice(a, a + int(rng.integers(1, 4))) for a in lo)] = rng.uniform(0.4, 1.0)
    f[-1, -1, -1] = 0.9
    return f


@pytest.mark.parametrize("dims", [(17, 33, 9), (2, 9, 41), (25, 25, 25), (64, 40, 18)], ids=str)
@pytest.mark.parametrize("values", ["sparse", "nan", "inf"])
@pytest.mark.parametrize("name,dt", DTYPES, ids=lambda d: str(d))
def test_leaps_over_empty_space_change_nothing(cuda_device, dims, values, name, dt):
    """Macro-cells are 8 cells wide: counts of cells that are and are not multiples
    of 8, and values that no range can bound."""
    s = dataclasses.replace(scenes.small(34, n=24, image=40, m=9, kind="noise", cutoff=0.99), dims=dims,
                            array=sparse(dims, sum(dims)))
    if values != "sparse":
        rng = np.random.default_rng(5)
        at = tuple(rng.integers(0, n, 6) for n in dims[::-1])
        s.array[at] = np.nan if values == "nan" else np.inf
    with renderer(s, dt) as r:
        r.set_tuning(light_brick=8, empty_skip=False, view_skip=False)
        ref = frame(r, s)
        for brick in (0, 8):
            r.set_tuning(light_brick=brick, empty_skip=True, view_skip=True)
            same(frame(r, s), ref, brick)
    if values == "sparse":
        o = oracle(s, name)
        om, _ = o.light_march()
        oimg, lit = o.view_march(om)
        assert np.array_equal(ref[1], om.ravel()) and ref[2][1] == lit
        check(ref[0], oimg)


def test_leaps_in_the_batched_form_change_nothing(cuda_device):
    s = [scenes.small(35 + i, n=24, image=40, m=9, kind="noise") for i in range(2)]
    dims = [(17, 33, 9), (41, 25, 24)]
    s = [dataclasses.replace(q, dims=d, array=sparse(d, 7)) for q, d in zip(s, dims)]
    with B.Renderer(0) as r:
        r.set_color_map(s[0].tf)
        r.batch_set_volumes([(q.array, q.origin, q.spacing, q.value_range) for q in s])
        ref = None
        for skip in (False, True):
            for split in (False, True):
                for brick in (0, 8, 16):
                    r.set_batch_options(light_brick=brick, skip=skip, split=split)
                    reqs = [r.request(i % 2, s[i % 2].camera(), light, kind, map_cells=7 + i,
                                      sample_distance=s[i % 2].sample_distance)
                            for i, (kind, light) in enumerate(LIGHTS)]
                    out, t = r.render_batch(reqs)
                    cur = out, (t["light_samples"], t["lit_samples"])
                    ref = ref or cur
                    assert cur[1] == ref[1], (skip, split, brick)
                    assert all(np.array_equal(a, b) for a, b in zip(out, ref[0])), (skip, split, brick)


@pytest.mark.parametrize("light", LIGHTS + [(0, (0.5, 2.0, 0.5)), (0, (-1.0, 0.5, 0.25)), (1, (0.0, -3.0, 0.0))],
                         ids=str)
def test_stitched_maps_for_lights_on_and_along_brick_faces(cuda_device, light):
    """Slab ratios of zero, without bound and undefined, where a product with the
    direction's reciprocal may not stand for the quotient."""
    s = dataclasses.replace(scenes.small(44, n=33, image=48, m=9, kind="noise"), dims=(33, 25, 29),
                            light_kind=light[0], light=light[1], array=None)
    bricks = scenes.split_bricks(s, (2, 3, 2))
    img, _, _, maps, lit = render_bricks(bricks)
    with B.Renderer(0) as r:
        bricks[0].configure(r)
        r.set_bricks([(b.field_numpy(), b.origin, b.spacing, b.value_range) for b in bricks])
        got, t = r.render(s.camera())
        assert t["lit_samples"] == lit
        for b in range(len(bricks)):
            assert np.array_equal(r.get_brick_map(b, 1, 1000), np.ravel(maps[b])), b
    check(got, img)


@pytest.mark.parametrize("nextra", [1, 3])
def test_several_lights_with_and_without_leaps(cuda_device, nextra):
    dims = (33, 20, 25)
    s = dataclasses.replace(scenes.small(36, n=24, image=48, m=9, kind="noise"), dims=dims, array=sparse(dims, 8))
    with renderer(s) as r:
        for kind, v in LIGHTS[:nextra]:
            (r.add_directional_light if kind else r.add_point_light)(v, (0.3, 0.9, 0.5), 0.7)
        r.set_multi_light(True)
        out = []
        for skip in (False, True):
            r.set_tuning(empty_skip=skip, view_skip=skip)
            img, t = r.render(s.camera())
            out.append((img, r.get_shadow_map((nextra + 1) * 1000), (t["light_samples"], t["lit_samples"])))
        same(out[1], out[0], "leaps")


@pytest.mark.parametrize("alpha", ["negative", "above one", "mixed"])
def test_colour_maps_outside_the_unit_range(cuda_device, alpha):
    """A negative opacity can take the accumulated one outside [0, 1], where the
    shaded colour has to be computed for every sample."""
    s = scenes.small(37, n=24, image=48, m=9, kind="blobs")
    s.tf = s.tf.copy()
    i = np.arange(len(s.tf))
    s.tf[:, 3] = {"negative": np.where(i % 7 == 0, -0.2, s.tf[:, 3]), "above one": s.tf[:, 3] * 3,
                  "mixed": np.where(i < 100, 0.0, np.where(i % 2, -0.6, 0.5))}[alpha]
    o = Oracle(s)
    om, _ = o.light_march()
    oimg, lit = o.view_march(om)
    with renderer(s) as r:
        for skip in (False, True):
            r.set_tuning(empty_skip=skip, view_skip=skip)
            img, m, n = frame(r, s)
            assert np.array_equal(m, om.ravel()) and n[1] == lit
            check(img, oimg)


# tiles of the field copy: 32 points along x, rows of y
COPY_DIMS = [(2, 2, 2), (3, 2, 33), (31, 3, 2), (32, 5, 4), (33, 4, 7), (34, 2, 3), (63, 3, 3), (64, 65, 2),
             (65, 2, 31), (129, 9, 5)]


@pytest.mark.parametrize("dims", COPY_DIMS, ids=str)
@pytest.mark.parametrize("name,dt", DTYPES, ids=lambda d: str(d))
def test_field_copy_at_every_remainder(cuda_device, dims, name, dt):
    s = scenes.small(38, n=24, image=24, m=5, kind="noise")
    rng = np.random.default_rng(sum(dims))
    s = dataclasses.replace(s, dims=dims, array=rng.uniform(0, 1, dims[::-1]).astype(np.float32))
    o = oracle(s, name)
    om, _ = o.light_march()
    oimg, lit = o.view_march(om)
    with renderer(s, dt) as r:
        img, m, n = frame(r, s)
        assert np.array_equal(m, om.ravel()) and n[1] == lit
        check(img, oimg)


# Spacing 1/32 and a step that divides it: sample after sample lands on a face, on
# an edge where two axes meet, and the middle ray of the odd image runs inside one.
@pytest.mark.parametrize("cam", [(0.5, 0.5, 2.0), (0.5, 2.0, 0.5), (-1.0, 0.5, 0.5), (2.0, 2.0, 0.5),
                                 (0.5, 0.5, 0.5)], ids=str)
@pytest.mark.parametrize("n", [33, 17])
def test_samples_on_cell_faces(cuda_device, cam, n):
    look = (0.5, 0.5, 0.5) if cam != (0.5, 0.5, 0.5) else (0.5, 0.5, 0.0)
    up = (1.0, 0.0, 0.0) if cam[0] == 0.5 else (0.0, 0.0, 1.0)
    s = dataclasses.replace(scenes.small(39, n=n, image=33, m=8, kind="noise"), cam_pos=cam, cam_look=look,
                            cam_up=up, sample_distance=1.0 / 64)
    rng = np.random.default_rng(3)  # faces where the value jumps: a wrong cell changes the pixel
    s.array = rng.uniform(0, 1, (n, n, n)).astype(np.float32)
    for light in ((1, (0.0, 0.0, -1.0)), (1, (1.0, 1.0, 0.0)), (0, (0.5, 0.5, 0.5))):
        s.light_kind, s.light = light
        o = Oracle(s)
        om, _ = o.light_march()
        oimg, lit = o.view_march(om)
        with renderer(s) as r:
            for skip in (False, True):
                r.set_tuning(empty_skip=skip, view_skip=skip)
                img, m, k = frame(r, s)
                assert np.array_equal(m, om.ravel()) and k[1] == lit, (light, skip)
                check(img, oimg)


@pytest.mark.parametrize("origin,spacing,cells", [(-3.7, 0.013, 200), (1000.0, 0.5, 64), (0.0, 1.0, 100),
                                                  (0.1, 3.0, 333), (-2.5e4, 7.7, 512), (0.0, 1e-20, 40),
                                                  (0.0, 1e20, 40), (5.0, 1e-6, 200)])
def test_cell_division_equals_ieee_at_any_scale(cuda_device, origin, spacing, cells):
    """Including widths past the range the two-term reciprocal is proven for, and
    cells whose rounded widths differ or vanish."""
    checked, bad = B.selftest_division(origin, spacing, cells, 1 << 12)
    assert checked > 0 and bad == 0


@pytest.mark.parametrize("kind", ["jitter", "power6", "one wide cell"])
@pytest.mark.parametrize("name,dt", DTYPES, ids=lambda d: str(d))
def test_coordinate_searches_from_both_starts(cuda_device, kind, name, dt):
    """Coordinates near their mean spacing are searched from its guess, others by halves."""
    s = scenes.small(40, n=40, image=40, m=9, kind="noise")
    n = s.dims[0]
    t = np.linspace(0.0, 1.0, n)
    wide = np.concatenate([t[:-1] * 1e-2, [1.0]])
    s.coords = {"jitter": stretched(n, "jitter", 4), "power6": (np.float32(t ** 6), np.float32(t), np.float32(1 - (1 - t) ** 2.5)),
                "one wide cell": tuple(np.float32(c) for c in (wide, t, wide))}[kind]
    o = oracle(s, name)
    om, _ = o.light_march()
    oimg, lit = o.view_march(om)
    with renderer(s, dt) as r:
        img, m, k = frame(r, s)
        assert np.array_equal(m, om.ravel()) and k[1] == lit
        check(img, oimg)


@pytest.mark.parametrize("n", [1, 2, 127, 129, 255, 257])
def test_network_features_by_pairs(cuda_device, n):
    """Bar: one bfloat16 ulp plus the phase error of a float32 position at 128 half-cycles."""
    s = scenes.small(81, n=24, image=16, m=8)
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    lf = rng.normal(size=(n, 3)).astype(np.float32)
    with renderer(s) as r:
        got = r.mlp_encode(pos, lf)
    ref = M.bf16(M.encode(pos, lf, (0, 0, 0), (1, 1, 1)))
    assert np.all(np.abs(got - ref) <= np.abs(ref) * 2.0 ** -7 + 1e-3)


@pytest.mark.parametrize("n", [127, 129, 148 * 128, 148 * 128 + 1, 6 * 148 * 128 + 5])
def test_dense_forward_around_its_tile_rounds(cuda_device, n):
    """Tiles are dealt to the CTAs' first pipelines, then their second, ...: one tile, a full
    round of first pipelines, one more, all six and a partial one. Bar: the rows' T equal the
    training kernel's, which deals its tiles otherwise, bit for bit (the same operations)."""
    s = scenes.small(83, n=24, image=16, m=8)
    rng = np.random.default_rng(n)
    with renderer(s) as r:
        r.mlp_set_params(rng.normal(0, 0.15, M.N_PARAMS).astype(np.float32))
        X = np.tile(rng.normal(0, 0.5, (1009, 112)).astype(np.float32), (n // 1009 + 1, 1))[:n]  # prime: no tile repeats
        T = r.mlp_forward_tc(X)
        _, _, T_train = r.mlp_loss_grad(X, np.zeros(n, np.float32))
    assert np.all(np.isfinite(T)) and np.array_equal(T, T_train)
    assert np.array_equal(T[1009:], T[:-1009] if n > 1009 else T[1009:])


@pytest.mark.parametrize("batch", [256, 512])
def test_overlapped_training_steps_follow_the_separate_ones(cuda_device, batch):
    """The step's two launches overlap their starts; the CUDA-core path runs whole launches
    one after the other. Bar: the held-out error after one epoch within 2% of the first
    error, the bound on the two backward passes' relative difference per step."""
    s = scenes.small(84, n=24, image=16, m=8)
    out = []
    for tensor in (True, False):
        with renderer(s) as r:
            r.mlp_set_tensor_cores(tensor)
            rep = r.mlp_train(B.mlp_options(samples_log2=14, epochs=1, batch=batch, lr=1e-3))
            out.append((rep["initial_rmse"], rep["holdout_rmse"]))
    assert out[0][1] < out[0][0]
    assert abs(out[0][1] - out[1][1]) <= 0.02 * out[1][0]


def test_training_buffers_kept_between_sizes(cuda_device):
    """The training set's buffers are kept up to 256 MB: a smaller set, a larger one
    that is given back, and the first again. Bar: the same seed's loss; the sums'
    order varies (2^-24 per addition, some hundred of them a weight and step), which 16
    steps at the step size 1e-3 keep below 1% of the error."""
    s = scenes.small(82, n=24, image=16, m=8)
    with renderer(s) as r:
        def rmse(log2):
            rep = r.mlp_train(B.mlp_options(samples_log2=log2, epochs=1, batch=1 << (log2 - 4), lr=1e-3))
            assert np.all(np.isfinite(r.mlp_params())) and rep["holdout_rmse"] < rep["initial_rmse"]
            return rep["holdout_rmse"]
        first = rmse(15)
        rmse(21)
        rmse(13)
        again = rmse(15)
    assert abs(again - first) <= 0.01 * first
