"""The choice among a principled surface's lobes where its random number is
exactly zero: the first lobe of the set, whatever ran on the GPU before."""
import numpy as np
import pytest

import oracle
from vision_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('spectrum', [2, 3, 4, 'srgb'])
def test_zero_lobe_choice_takes_the_first_lobe(vb, gpu_ctx, spectrum):
    # One of the 12 paths of pixel (99, 109) draws a zero there, on a surface
    # without a sheen lobe.
    sc = scenes.principled_room(width=160, height=120, max_depth=8, dimension=3 if spectrum == 'srgb' else spectrum)
    if spectrum == 'srgb':
        sc['spectrum'] = {'type': 'srgb'}
    s = vb.Scene(gpu_ctx, sc).build_accel()
    want = oracle.OracleScene(s).paths(np.array([99 * 160 + 109], np.uint32), 0, 12)[:, 0].mean(0)
    other = vb.Scene(gpu_ctx, scenes.material_room(width=160, height=120)).build_accel()
    films = []
    for schedule in ('grid', 'persistent', 'wavefront', 'wavefront_binned'):
        s.set_schedule(schedule)
        for _ in range(2):
            s.render(0, 12)
            films.append(s.film())
            other.render(0, 3)
    assert all(np.array_equal(films[0], f) for f in films[1:])
    assert np.all(np.abs(films[0][99, 109, :3] - want) <= 1e-3 * (1.0 + np.abs(want)))
