"""vs_render's default schedule ('auto') on both sides of the size where it
changes from the persistent megakernel to wavefront passes, and wavefront
passes across waves: the film is the same bits as from schedules that take one
form at every size."""
import copy

import numpy as np
import pytest

from helpers import write_room_textures
from vision_b200 import scenes

pytestmark = pytest.mark.gpu

# Paths up to which the megakernel renders, per bounce of depth (at most 16).
DIFFUSE, OTHER = 7168, 1536


def _films(vb, ctx, sc, frames, schedules, fp64=False):
    s = vb.Scene(ctx, sc).build_accel()
    out = []
    for schedule in schedules:
        s.set_schedule(schedule)
        s.render(0, frames, fp64=fp64)
        out.append((s.film(), s.film(vb.FILM_SUM64) if fp64 else None))
    return out


ROOMS = {
    'box': (scenes.box_room, DIFFUSE), 'material': (scenes.material_room, OTHER),
    'substrate': (scenes.substrate_room, OTHER), 'plastic': (scenes.plastic_room, OTHER),
    'principled': (scenes.principled_room, OTHER), 'metallic': (scenes.metallic_room, OTHER),
    'point': (scenes.point_light_room, DIFFUSE),
}


@pytest.mark.parametrize('depth', [1, 2, 8])
@pytest.mark.parametrize('room', sorted(ROOMS))
def test_film_on_both_sides_of_the_line(vb, gpu_ctx, room, depth):
    make, per_depth = ROOMS[room]
    line = min(depth, 16) * per_depth
    w = 97
    h = -(-line // (4 * w))
    sc = make(width=w, height=h, max_depth=depth, dimension=3 + depth % 2)
    for frames in (3, 4, 5):  # below, just above and above the line
        (grid, _), (waves, _), (film, _) = _films(vb, gpu_ctx, sc, frames, ['grid', 'wavefront', 'auto'])
        assert np.array_equal(grid, film), (frames, w * h * frames, line)
        assert np.array_equal(waves, film), (frames, w * h * frames, line)
        assert film[..., :3].max() > 0.0


@pytest.mark.parametrize('room', ['box', 'principled'])
def test_named_schedules_keep_their_form(vb, gpu_ctx, room):
    # The grid and the megakernel are one kernel and the film pass; wavefront
    # passes are several for each bounce, at any size.
    s = vb.Scene(gpu_ctx, ROOMS[room][0](width=16, height=16, max_depth=4)).build_accel()
    count = {}
    for schedule in (None, 'grid', 'persistent', 'wavefront', 'wavefront_binned', 'auto'):
        if schedule:
            s.set_schedule(schedule)
        n = vb.launch_count()
        s.render(0, 1)
        count[schedule] = vb.launch_count() - n
    assert count[None] == count['auto'] == count['persistent'] == count['grid'] == 2
    assert count['wavefront'] >= 2 + 2 * 4
    assert count['wavefront_binned'] > count['wavefront']


@pytest.mark.parametrize('dimension', [1, 2, 3, 4])
def test_environment_scene_in_wavefront_form(vb, gpu_ctx, dimension):
    sc = scenes.large_scene(width=120, height=101, max_depth=12, subdivisions=3, grid=40, tiles=4, sky_width=256,
                            sky_height=128, dimension=dimension)
    assert 120 * 101 * 3 > 12 * OTHER
    # (At one wavelength the megakernel rounds the microfacet lobes differently.)
    others = ['wavefront_binned', 'auto'] + ([] if dimension == 1 else ['grid', 'persistent'])
    for frames in (1, 3):
        films = _films(vb, gpu_ctx, sc, frames, ['wavefront'] + others, fp64=True)
        for film, sums in films[1:]:
            assert np.array_equal(films[0][0], film)
            assert np.array_equal(films[0][1], sums)


def test_two_level_scene_in_wavefront_form(vb, gpu_ctx):
    sc = scenes.instanced_scene(width=150, height=110, copies=9, subdivisions=4, patch=30, max_depth=10)
    sc['render_setting']['instancing'] = True
    (grid, _), (film, _), (auto, _) = _films(vb, gpu_ctx, sc, 2, ['grid', 'wavefront', 'auto'])
    assert 150 * 110 * 2 > 10 * OTHER
    assert np.array_equal(grid, film)
    assert np.array_equal(grid, auto)


@pytest.mark.parametrize('frames', [1, 2])
@pytest.mark.parametrize('room', sorted(ROOMS))
def test_rgb_spectrum(vb, gpu_ctx, room, frames):
    sc = ROOMS[room][0](width=160, height=100)
    sc.pop('spectrum')
    (binned, _), (film, _), (auto, _) = _films(vb, gpu_ctx, sc, frames, ['wavefront_binned', 'wavefront', 'auto'])
    assert np.array_equal(binned, film)
    assert np.array_equal(auto, film)


@pytest.mark.parametrize('room', sorted(ROOMS))
def test_one_wavelength(vb, gpu_ctx, room):
    sc = ROOMS[room][0](width=90, height=60, dimension=1)
    (binned, _), (film, _), (auto, _) = _films(vb, gpu_ctx, sc, 1, ['wavefront_binned', 'wavefront', 'auto'])
    assert np.array_equal(binned, film)
    assert np.array_equal(auto, film)


def test_film_across_waves(vb, gpu_ctx):
    # 17 x 2^20 paths: one full wave of 2^24 path slots and a second, smaller
    # one; five waves of the binned schedule.
    sc = scenes.box_room(width=1024, height=1024, max_depth=5)
    (grid, _), (film, _), (binned, _) = _films(vb, gpu_ctx, sc, 17, ['grid', 'wavefront', 'wavefront_binned'])
    assert np.array_equal(grid, film)
    assert np.array_equal(grid, binned)


def _lens(sc):
    sc['camera']['type'] = 'thin_lens'
    sc['camera']['param'].update(lens_radius=0.02, focal_distance=1.2)
    sc['camera']['param']['filter'] = {'type': 'mitchell', 'param': {'radius': [2.0, 2.0]}}
    return sc


def _instanced(**kw):
    sc = scenes.instanced_scene(copies=9, subdivisions=4, patch=30, **kw)
    sc['render_setting']['instancing'] = True
    return sc


def _outdoors(**kw):
    return scenes.large_scene(subdivisions=3, grid=40, tiles=4, sky_width=256, sky_height=128, **kw)


def _diffuse_outdoors(**kw):
    sc = _outdoors(**kw)
    diffuse = next(m for m in scenes.box_room()['materials'] if m['type'] == 'diffuse')
    sc['materials'] = [m if m['type'] == 'black_body' else dict(copy.deepcopy(diffuse), name=m['name'])
                       for m in sc['materials']]
    return sc


FORMS = dict({k: v[0] for k, v in ROOMS.items()}, textured=scenes.textured_room, projector=scenes.projector_room,
             lens=lambda **kw: _lens(scenes.box_room(**kw)), material_lens=lambda **kw: _lens(scenes.material_room(**kw)),
             outdoors=_outdoors, diffuse_outdoors=_diffuse_outdoors, instanced=_instanced)


@pytest.mark.parametrize('dimension', [1, 2, 3, 4, 'srgb'])
@pytest.mark.parametrize('form', sorted(FORMS))
def test_split_renders_and_forms_agree(vb, gpu_ctx, tmp_path, form, dimension):
    # One render call above the line and calls of one frame below it give the
    # same film, that of the wavefront passes.
    write_room_textures(str(tmp_path))
    sc = FORMS[form](width=101, height=79, max_depth=8, **({} if dimension == 'srgb' else {'dimension': dimension}))
    if dimension == 'srgb':
        sc['spectrum'] = {'type': 'srgb'}
    s = vb.Scene(gpu_ctx, sc, base_dir=str(tmp_path)).build_accel()
    frames = 8
    assert 101 * 79 <= 8 * OTHER and 101 * 79 * frames > 8 * DIFFUSE
    s.set_schedule('wavefront')
    s.render(0, frames)
    want = s.film()
    s.set_schedule('auto')
    s.render(0, frames)
    assert np.array_equal(s.film(), want)
    for f in range(frames):
        s.render(f, 1)
    assert np.array_equal(s.film(), want)
