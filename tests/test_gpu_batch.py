"""Batch configuration through the C ABI: the autotuner (rmn_batch_autotune),
the memory query it caps candidates with (rmn_batch_device_bytes), and the
library's default unit split, which must be a choice of each render alone.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from raym0nade_gb300 import _lib, api, scenes  # noqa: E402

SLOTS, POOLS, LANES, STACKS = {0, 2, 4, 8, 16}, {0, 1 << 20, 1 << 21, 1 << 22, 1 << 23}, {0, 2, 3, 4}, {23, 27}


def _photo_np(ph):
    return [x.cpu().numpy() for x in (ph.radiance_Dd, ph.radiance_Ds, ph.radiance_Id, ph.radiance_Is, ph.Gbuffer)]


def _uneven_items():
    """Four renders of uneven size: Cornell boxes, a heightfield under a sky,
    a triangle soup."""
    cor = api.Model(scenes.cornell())
    hf = scenes.heightfield(48, seed=2, extent=4.8, patch=8)
    hf.env = scenes.sky_env(64, 32, sun_radiance=100.0, sun_diameter_deg=8.0)
    sky = api.Model(hf)
    soup = api.Model(scenes.random_soup(20000, 5))
    skycam = scenes.Camera((0.3, 2.0, -0.8), (0.35, -0.45, 0.82), (0.0, -1.0, 0.0), (-1.0, 0.0, 0.0), 0.02, 96, 64, 24)
    specs = [(cor, scenes.cornell_camera(128, 128, 32), 1), (sky, skycam, 2),
             (cor, scenes.cornell_camera(64, 80, 12, max_depth=6), 3), (soup, scenes.soup_camera(96, 96, 16, 8), 4)]
    return [(m, api.RenderArgs.from_camera(c, seed=s), api.Photo(c.width, c.height)) for m, c, s in specs]


def _free_bytes():
    free, _ = torch.cuda.mem_get_info()
    return free


def test_autotune_returns_a_candidate_and_its_images_match():
    items = _uneven_items()
    free = _free_bytes()
    res = api.autotune(items, pixel_fraction=0.25)
    assert res["slots_per_unit"] in SLOTS and res["pool_workers"] in POOLS and res["lanes"] in LANES
    assert res["stack_entries"] in STACKS and res["ray_order"] in (0, 1)
    # these trees are shallow: both stack builds are admissible, the shallow
    # one is the default and the deeper one is timed once more; then binned
    # ray queues
    assert res["candidates"] >= 3
    assert 0.0 < res["best_ms"] <= res["default_ms"]
    # the choice fits the tuner's memory cap: half of the free device memory
    for m, a, ph in items:
        a.slots_per_unit = res["slots_per_unit"]
    assert api.batch_device_bytes(items, res["pool_workers"], res["lanes"]) <= free // 2
    # a batch built with the tuned settings renders every item exactly as
    # rmn_render does with the same slots per unit
    b = api.Batch(items, use_graph=True, pool_workers=res["pool_workers"], lanes=res["lanes"],
                  stack_entries=res["stack_entries"], ray_order=res["ray_order"])
    b.render()
    torch.cuda.synchronize()
    for m, a, ph in items:
        for x, y in zip(_photo_np(ph), _photo_np(api.render(m, a))):
            assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("use_graph", [True, False])
def test_stack_builds_and_ray_order_give_identical_images(use_graph):
    """Both traversal stack builds, with and without binned ray queues, give
    every item exactly its rmn_render images (twice in a row)."""
    items = _uneven_items()
    solo = [_photo_np(api.render(m, a)) for m, a, _ in items]
    for stack in (23, 27):
        for order in (0, 1):
            b = api.Batch(items, use_graph=use_graph, stack_entries=stack, ray_order=order, lanes=2)
            for _ in range(2):
                b.render()
                torch.cuda.synchronize()
                for (m, a, ph), ref in zip(items, solo):
                    for x, y in zip(_photo_np(ph), ref):
                        assert np.array_equal(x, y, equal_nan=True)
    with pytest.raises(api.RmnError) as e:
        api.Batch(items, stack_entries=24)
    assert e.value.status == 1
    with pytest.raises(api.RmnError) as e:
        api.Batch(items, ray_order=2)
    assert e.value.status == 1


def test_device_bytes_counts_units_and_workers():
    items = _uneven_items()[:1]  # 128 x 128 Cornell, 32 spp
    m, a, ph = items[0]
    a.slots_per_unit = 4
    # light-sample slots in units of max(4, 8), path slots in units of 4
    spp_d = int(32 * 0.7)
    units = 128 * 128 * ((spp_d + 7) // 8 + (32 - spp_d + 3) // 4)
    one = api.batch_device_bytes(items, 128, 1)
    two = api.batch_device_bytes(items, 256, 1)
    per_worker = (two - one) / 128
    assert 500 < per_worker < 1200
    assert one == units * 112 + 128 * per_worker
    # the pool never exceeds one worker per unit
    assert api.batch_device_bytes(items, 1 << 23, 1) == units * 112 + units * per_worker


def test_autotune_rejects_an_impossible_budget():
    """A batch whose unit records alone exceed the free device memory: the
    tuner reports RMN_ERR_OUT_OF_MEMORY instead of a configuration."""
    m = api.Model(scenes.cornell())
    cam = scenes.cornell_camera(1024, 1024, 1024)
    a = api.RenderArgs.from_camera(cam, seed=1)
    a.slots_per_unit = 1
    items = [(m, a, api.Photo(8, 8))]
    need = api.batch_device_bytes(items, 4096, 1)
    _lib.load().rmn_release_cached_memory()
    torch.cuda.empty_cache()
    free = _free_bytes()
    filler = None
    if need < free:
        filler = torch.empty(free - need // 2, dtype=torch.uint8, device="cuda")
    with pytest.raises(api.RmnError) as e:
        api.autotune([(m, a, api.Photo(cam.width, cam.height))], pixel_fraction=1.0 / 64)
    assert e.value.status == 3  # RMN_ERR_OUT_OF_MEMORY
    del filler
    torch.cuda.empty_cache()
    with pytest.raises(api.RmnError) as e:
        api.autotune(_uneven_items(), pixel_fraction=0.0)
    assert e.value.status == 1


def test_default_split_depends_on_the_render_alone():
    """The library's default unit split (slots_per_unit = 0) decides the
    float summation order of a pixel's samples, so it must not change with
    the free device memory or the batch around a render: the same render
    with most of the device memory taken, and inside a batch, is
    bit-identical."""
    m = api.Model(scenes.cornell())
    cam = scenes.cornell_camera(512, 512, 256)  # 2^26 sample slots: 33.5 M units of 112 B at 2 slots
    a = api.RenderArgs.from_camera(cam, seed=8)
    ref = _photo_np(api.render(m, a))
    _lib.load().rmn_release_cached_memory()
    torch.cuda.empty_cache()
    free = _free_bytes()
    keep = 12 << 30  # the unit records (3.75 GB) exceed a quarter of what is left
    filler = torch.empty(max(free - keep, 1), dtype=torch.uint8, device="cuda") if free > keep else None
    got = _photo_np(api.render(m, a))
    del filler
    torch.cuda.empty_cache()
    for x, y in zip(got, ref):
        assert np.array_equal(x, y, equal_nan=True)
    other = _uneven_items()
    ph = api.Photo(cam.width, cam.height)
    b = api.Batch([(m, a, ph)] + other, use_graph=True)
    b.render()
    torch.cuda.synchronize()
    for x, y in zip(_photo_np(ph), ref):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("lanes", [0, 1, 3])
def test_device_bytes_of_a_batch_of_few_units(lanes):
    """256 x 256 at 16 spp, 5 units a pixel: rendered on one lane with at most
    1024 workers per SM, whatever the pool and the lanes asked for, and
    rmn_batch_device_bytes counts those."""
    m = api.Model(scenes.cornell())
    a = api.RenderArgs.from_camera(scenes.cornell_camera(256, 256, 16), seed=1)
    items = [(m, a, api.Photo(256, 256))]
    units = 256 * 256 * 5
    held = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    one, two = (api.batch_device_bytes(items, n, 1) for n in (128, 256))
    per_worker = (two - one) / 128
    assert held < units
    assert api.batch_device_bytes(items, 0, lanes) == units * 112 + held * per_worker
    assert api.batch_device_bytes(items, 1 << 20, lanes) == units * 112 + held * per_worker
    assert api.batch_device_bytes(items, 1000, lanes) == units * 112 + 1000 * per_worker


@pytest.mark.parametrize("spp,direct", [(1, True), (4, True), (8, False), (64, False), (4096, False)])
def test_few_units_of_many_slots_are_much_work(spp, direct):
    """A render of one unit a pixel and 2000 units per SM: it goes without the
    wavefront, on 1024 workers per SM, only while its sample slots would make no
    more than 4000 units of two (the light samples: of eight) per SM; with
    glass, whatever their number."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w = int((2000 * sms) ** 0.5)
    spp_d = int(np.float32(spp) * np.float32(0.7))
    assert direct == (w * w * ((spp_d + 7) // 8 + (spp - spp_d + 1) // 2) <= 4000 * sms)
    for scene, held in ((scenes.cornell(), 1024 * sms if direct else w * w), (scenes.cornell_glass(), 1024 * sms)):
        a = api.RenderArgs.from_camera(scenes.cornell_camera(w, w, spp), lanes_per_pixel=1)
        items = [(api.Model(scene), a, api.Photo(8, 8))]
        full, one, two = (api.batch_device_bytes(items, n, 1) for n in (1 << 20, 128, 256))
        assert full == one + (held - 128) * (two - one) // 128


def test_autotune_times_what_differs():
    """A batch rendered without the wavefront differs by its slots per unit and
    its stack alone: the library's choice, four splits and the deeper stack."""
    res = api.autotune(_uneven_items(), pixel_fraction=0.25)
    assert res["candidates"] == 6 and res["ray_order"] == 0


def _large_items(kind):
    """Renders of some 425,000 units in all, above the line under which a
    batch is rendered without the wavefront; `alpha`: one with cut-outs, whose
    shadow rays are searched in order, and one with glass."""
    hf = scenes.heightfield(120, seed=2, extent=12.0, patch=8)
    hf.env = scenes.sky_env(64, 32, sun_radiance=100.0, sun_diameter_deg=8.0)
    skycam = scenes.Camera((0.3, 2.0, -0.8), (0.35, -0.45, 0.82), (0.0, -1.0, 0.0), (-1.0, 0.0, 0.0), 0.01, 192, 128, 12)
    specs = [(scenes.cornell(), scenes.cornell_camera(224, 224, 16), 1), (hf, skycam, 2)]
    if kind == "alpha":
        specs += [(scenes.textured_room(), scenes.textured_camera(160, 96, 12), 3),
                  (scenes.cornell_glass(), scenes.cornell_camera(64, 48, 4), 4)]
    else:
        specs += [(scenes.random_soup(20000, 5), scenes.soup_camera(160, 128, 16, 8), 5)]
    return [(api.Model(s), api.RenderArgs.from_camera(c, seed=k), api.Photo(c.width, c.height)) for s, c, k in specs]


@pytest.mark.parametrize("lanes", [1, 2, 3])
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("kind", ["plain", "alpha"])
def test_wavefront_batches_give_identical_images(kind, use_graph, lanes):
    """The wavefront with one lane (its launches overlapped, also inside a
    captured graph) and with several, both traversal stack builds, with and
    without binned ray queues, its end in block_kernel, and new arguments for a
    built batch: every item's images are those of the wavefront alone, which
    rmn_render_profile_get renders with."""
    import dataclasses
    items = _large_items(kind)
    units = (api.batch_device_bytes(items, 128, 1) - 128 * 1300) // 112
    assert units > 2632 * torch.cuda.get_device_properties(0).multi_processor_count
    moved = [dataclasses.replace(a, seed=a.seed + 20) for _, a, _ in items]
    want = [[_photo_np(api.render_profile(m, b)[0]) for (m, _, _), b in zip(items, args)]
            for args in ([a for _, a, _ in items], moved)]
    for stack in (23, 27):
        for order in (0, 1):
            b = api.Batch(items, use_graph=use_graph, stack_entries=stack, ray_order=order, lanes=lanes)
            for k in (0, 0, 1):
                b.update([a for _, a, _ in items] if k == 0 else moved)
                b.render()
                torch.cuda.synchronize()
                for (_, _, ph), ref in zip(items, want[k]):
                    for x, y in zip(_photo_np(ph), ref):
                        assert np.array_equal(x.view(np.int32), y.view(np.int32)), (stack, order, k)
