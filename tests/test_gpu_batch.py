"""Batched tracing (qmcrt_batch_*) against the plain path, on the GPU.

A batch instance (scene, sun) must behave exactly like the plain scene after
qmcrt_scene_set_sun(sun): the device-prepared geometry is bit-identical to
the host's, and in the exact math mode per-ray outcomes are identical, so
flux images agree up to the order of float atomic accumulation
(L1 <= 1e-5) and FP64 powers up to summation order (<= 1e-9 relative).
"""
import numpy as np
import pytest

import solarenergy_chier_b200 as q
from solarenergy_chier_b200 import synth

pytestmark = pytest.mark.gpu

SUNS = [[0.0, -0.866, -0.5], [0.35, -0.75, 0.56], [-0.5, -0.6, 0.62]]


@pytest.fixture(scope="module")
def fields(tmp_path_factory, cuda_device):
    big = synth.large_field(tmp_path_factory.mktemp("b1"), seed=6, num_heliostats=24, helio_pixel=0.25,
                            receiver_pixel=0.05, groups=4, per_group=128)
    small = synth.small_field(tmp_path_factory.mktemp("b2"), seed=2, helio_pixel=0.2, groups=4, per_group=128)
    return big, small


def scenes_of(fields):
    return [q.Scene(f.scene, f.config, device=0, seed=11) for f in fields]


def plain_reference(f, sun, mode):
    s = q.Scene(f.scene, f.config, device=0, seed=11)
    s.set_sun(sun)
    s.set_math_mode(mode)
    s.trace(list(range(s.num_heliostats)))
    per, total = s.power()
    return s, s.image(0), per, total


def test_device_preparation_equals_host(fields):
    scenes = scenes_of(fields)
    inst = [(0, SUNS[0]), (0, SUNS[1]), (1, SUNS[2]), (1, SUNS[0])]
    b = q.Batch(scenes, inst)
    for k, (si, sun) in enumerate(inst):
        ref = q.Scene(fields[si].scene, fields[si].config, device=-1)
        ref.set_sun(sun)
        verts, normals = b.geometry(k, 0)
        assert np.array_equal(verts, ref.grid(0)["vertices"]), f"instance {k}: vertices differ"
        want = np.stack([ref.heliostat(h)["normal"] for h in range(ref.num_heliostats)])
        assert np.array_equal(normals, want), f"instance {k}: normals differ"


@pytest.mark.parametrize("mode", [1, 0])
def test_batch_equals_plain_per_sun(fields, mode):
    scenes = scenes_of(fields)
    inst = [(0, SUNS[0]), (0, SUNS[1]), (1, SUNS[2]), (1, SUNS[1])]
    b = q.Batch(scenes, inst)
    b.set_math_mode(mode)
    b.trace()
    for k, (si, sun) in enumerate(inst):
        _, img, per, total = plain_reference(fields[si], sun, mode)
        got = b.image(k).astype(np.float64)
        l1 = np.abs(got - img).sum() / img.sum()
        assert l1 <= 1e-5, f"instance {k}: flux L1 {l1:.2e}"
        gper, gtotal = b.power(k)
        assert abs(gtotal - total) <= 1e-9 * total
        assert np.allclose(gper, per, rtol=1e-9, atol=0)


def test_graph_replay_and_set_suns(fields):
    scenes = scenes_of(fields)
    inst = [(0, SUNS[0]), (1, SUNS[1])]
    b = q.Batch(scenes, inst)
    b.set_math_mode(1)
    b.set_light_range(0, 64)
    b.trace()
    first = [b.image(k) for k in range(2)]
    b.capture_graph(clear_first=True)
    b.graph_launch()
    b.graph_launch()  # clears, then traces again: same images
    for k in range(2):
        assert np.abs(b.image(k) - first[k]).sum() <= 1e-5 * first[k].sum()
    # new suns prepared on the device equal a plain scene with those suns
    b.set_suns([SUNS[2], SUNS[0]])
    b.clear()
    b.set_light_range(0, 128)
    b.trace()
    for k, (si, sun) in enumerate([(0, SUNS[2]), (1, SUNS[0])]):
        _, img, _, total = plain_reference(fields[si], sun, 1)
        assert np.abs(b.image(k) - img).sum() <= 1e-5 * img.sum()
        assert abs(b.power(k)[1] - total) <= 1e-9 * total


def test_autotune_and_errors(fields):
    scenes = scenes_of(fields)
    b = q.Batch(scenes, [(0, SUNS[0]), (1, SUNS[1])])
    shape, ms = b.autotune()
    assert 0 <= shape < len(q.launch_shapes()) and len(ms) == len(q.launch_shapes()) and min(ms) > 0
    assert ms[shape] == min(ms)
    assert b.power(0)[1] == 0.0  # autotune clears
    with pytest.raises(q.QmcrtError):
        b.set_light_range(0, 10 ** 6)
    with pytest.raises(q.QmcrtError):
        b.image(5)
    with pytest.raises(q.QmcrtError):
        b.graph_launch()
    with pytest.raises(q.QmcrtError):
        q.Batch(scenes, [(2, SUNS[0])])
    with pytest.raises(q.QmcrtError):
        q.Batch(scenes, [(0, [0.0, 0.0, 0.0])])


def test_uneven_fields_batch_equals_plain(tmp_path):
    """Two of the batch benchmark's uneven fields (a rectangle receiver with
    flat heliostats, a cylinder with focus-flat ones), coarse facets, at
    their own suns and at a shared one, in one batch with mismatched sizes."""
    files = [synth.uneven_field(tmp_path, k, seed=3, helio_pixel=0.75, groups=4, per_group=128) for k in (0, 1)]
    scenes = [q.Scene(f.scene, f.config, device=0, seed=11) for f in files]
    own = [np.array(s.info.sun_dir[:], np.float32) for s in scenes]
    inst = [(0, own[0]), (1, own[1]), (1, SUNS[1]), (0, SUNS[2])]
    b = q.Batch(scenes, inst)
    b.set_math_mode(1)
    b.trace()
    for k, (si, sun) in enumerate(inst):
        _, img, per, total = plain_reference(files[si], sun, 1)
        assert total > 0, f"instance {k}: no energy"
        got = b.image(k).astype(np.float64)
        assert np.abs(got - img).sum() <= 1e-5 * img.sum(), f"instance {k}"
        gper, gtotal = b.power(k)
        assert abs(gtotal - total) <= 1e-9 * total
        assert np.allclose(gper, per, rtol=1e-9, atol=0)


@pytest.mark.parametrize("heliostats,lights", [(1, 1), (1, 37), (3, 33), (1, 994), (1, 995), (50, 199), (50, 200)])
def test_chunk_sizes_of_small_launches(heliostats, lights, tmp_path):
    """Flux launches below 6.4 M and 64 M rays take 8- and 16-iteration warp
    chunks; either side of both limits (and chunks that end inside a facet)
    they give what 64-iteration chunks of another launch shape do: the same
    flux up to float atomic order (L1 <= 1e-6) and FP64 powers (1e-12)."""
    f = synth.small_field(tmp_path, seed=1)
    s = q.Scene(f.scene, f.config, device=0, seed=2)
    s.set_light_range(5, 5 + lights)
    ids = list(range(heliostats))
    out = []
    for shape in (3, 0):  # two-warp blocks of 64-iteration chunks, then the default shape
        s.set_launch_shape(shape)
        s.clear()
        s.clear_power()
        s.trace(ids)
        out.append((s.image(0).astype(np.float64), s.power()[0]))
    (img0, p0), (img, p) = out
    assert p0.sum() > 0 and np.abs(img - img0).sum() <= 1e-6 * img0.sum()
    np.testing.assert_allclose(p, p0, rtol=1e-12, atol=0)


@pytest.mark.parametrize("mode", [0, 1])
def test_spread_images_of_small_receivers(mode, tmp_path):
    """Flux launches of 1.5 M rays and more onto small receivers deposit
    into spread images: one launch gives what smaller launches over the same
    lights add up to directly (L1 <= 1e-6, FP64 powers 1e-12), on both
    receivers of a scene, a second launch adds to the images, and nothing is
    left in the spread ones."""
    f = synth.two_receiver_field(tmp_path, seed=1, helio_pixel=0.05, groups=4, per_group=128)
    s = q.Scene(f.scene, f.config, device=0, seed=2)
    s.set_math_mode(mode)
    ids = list(range(s.num_heliostats))
    facets = sum(s.heliostat(h)["num_facets"] for h in ids)
    assert 4 * facets < 1.5e6 <= 12 * facets

    def traced(ranges):
        s.clear()
        s.clear_power()
        for r in ranges:
            s.set_light_range(*r)
            s.trace(ids)
        return [s.image(k).astype(np.float64) for k in (0, 1)], s.power()[0]

    pieces, p0 = traced([(3, 7), (7, 11), (11, 15)])
    for times in (1, 2):
        images, p = traced([(3, 15)] * times)
        for a, b in zip(images, pieces):
            assert b.sum() > 0 and np.abs(a - times * b).sum() <= 1e-6 * times * b.sum()
        np.testing.assert_allclose(p, times * p0, rtol=1e-12, atol=0)


@pytest.mark.parametrize("kind,pixel", [("small", 0.0345), ("small", 0.0344), ("two", 0.033)])
def test_spread_images_and_large_ones(kind, pixel, tmp_path):
    """Either side of the largest image that has a spread one, and a scene
    with one receiver on each side: lists of one receiver's heliostats and of
    both, one launch after another, give what another launch shape's direct
    deposits do (L1 <= 1e-5, FP64 powers 1e-12)."""
    make = synth.small_field if kind == "small" else synth.two_receiver_field
    f = make(tmp_path, seed=1, helio_pixel=0.05, receiver_pixel=pixel, groups=4, per_group=128)
    s = q.Scene(f.scene, f.config, device=0, seed=2)
    pixels = [s.receiver(r)["width"] * s.receiver(r)["height"] for r in range(s.num_receivers)]
    assert [n <= 40000 for n in pixels] == {0.0345: [True], 0.0344: [False], 0.033: [True, False]}[pixel]
    ids = list(range(s.num_heliostats))
    half = len(ids) // 2
    s.set_light_range(0, 24)
    out = []
    for shape in (3, 0):  # two-warp blocks never use spread images
        s.set_launch_shape(shape)
        s.clear()
        s.clear_power()
        for part in (ids, ids[:half], ids[half:], ids[::2]):
            s.trace(part)
        out.append(([s.image(r).astype(np.float64) for r in range(s.num_receivers)], s.power()[0]))
    for a, b in zip(out[1][0], out[0][0]):
        assert b.sum() > 0 and np.abs(a - b).sum() <= 1e-5 * b.sum()
    np.testing.assert_allclose(out[1][1], out[0][1], rtol=1e-12, atol=0)


@pytest.mark.parametrize("towers", [4, 5])
def test_spread_images_of_as_many_receivers_as_there_are(towers, tmp_path):
    """Scenes of four receivers have spread images, of five none: small
    receivers side by side, traced one after another and all at once, give what
    another launch shape's direct deposits do (L1 <= 1e-5, FP64 powers 1e-12)."""
    f = synth.small_field(tmp_path, seed=1, groups=4, per_group=128, rows=2, cols=4)
    lines = f.scene.read_text().splitlines()
    first = lines.index("Recv\t0")
    head, field = lines[:first], lines[first:]
    out = [line.replace("ngrid\t1", f"ngrid\t{towers}") for line in head]
    for k in range(towers):  # the same tower and field, 300 m further east
        for line in field:
            words = line.split()
            if words and words[0] in ("pos", "helio"):
                line = f"{words[0]}\t{float(words[1]) + 300.0 * k:.6f}\t{words[2]}\t{words[3]}"
            out.append(line)
    f.scene.write_text("\n".join(out) + "\n")
    s = q.Scene(f.scene, f.config, device=0, seed=2)
    assert s.num_receivers == towers and s.num_heliostats == 8 * towers
    s.set_light_range(0, 32)  # 1.6 M rays a tower
    images = []
    for shape in (3, 0):
        s.set_launch_shape(shape)
        s.clear()
        s.clear_power()
        for k in range(towers):
            s.trace(list(range(8 * k, 8 * k + 8)))
        s.trace(list(range(8 * towers)))
        images.append(([s.image(r).astype(np.float64) for r in range(towers)], s.power()[0]))
    for a, b in zip(images[1][0], images[0][0]):
        assert b.sum() > 0 and np.abs(a - b).sum() <= 1e-5 * b.sum()
    np.testing.assert_allclose(images[1][1], images[0][1], rtol=1e-12, atol=0)


def test_every_launch_shape_gives_the_same_result(fields, tmp_path):
    """The autotuner's candidates (launch shapes of the production build:
    block widths, warp chunks of 32, 64 or 128 iterations) change only how
    rays are handed to warps: every shape gives the same flux (up to float
    atomic order, L1 <= 1e-6) and FP64 powers (1e-12) on a plain scene and
    on a batch, with ragged light counts (37 lights: warps span facets and
    chunks end inside one), and the plain autotuner keeps the fastest."""
    shapes = q.launch_shapes()
    assert shapes[0] == (32, 64, False) and len(shapes) >= 5 and any(x[2] for x in shapes)
    f = fields[1]
    s = q.Scene(f.scene, f.config, device=0, seed=4)
    ids = list(range(s.num_heliostats))
    s.set_light_range(3, 40)
    ref = None
    for k in range(len(shapes)):
        s.set_launch_shape(k)
        s.clear()
        s.clear_power()
        s.trace(ids)
        img = s.image(0).astype(np.float64)
        per, total = s.power()
        if ref is None:
            ref = (img, per, total)
            assert total > 0
            continue
        assert np.abs(img - ref[0]).sum() <= 1e-6 * ref[0].sum(), shapes[k]
        np.testing.assert_allclose(per, ref[1], rtol=1e-12, atol=0)
    best, ms = s.autotune(ids)
    assert ms[best] == min(ms) and min(ms) > 0
    assert s.power()[1] == 0.0
    s.trace(ids)  # the chosen shape traces like the others
    assert abs(s.power()[1] - ref[2]) <= 1e-12 * ref[2]
    scenes = scenes_of(fields)
    b = q.Batch(scenes, [(0, SUNS[0]), (1, SUNS[1])])
    b.set_light_range(1, 38)
    first = None
    for k in range(len(shapes)):
        b.set_launch_shape(k)
        b.clear()
        b.trace()
        out = [(b.image(i).astype(np.float64), b.power(i)[1]) for i in range(2)]
        if first is None:
            first = out
            continue
        for (img, tot), (img0, tot0) in zip(out, first):
            assert np.abs(img - img0).sum() <= 1e-6 * img0.sum()
            assert abs(tot - tot0) <= 1e-12 * tot0
