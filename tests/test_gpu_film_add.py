"""Splats into a caller's film: one bulk reduction per splat where the film is 16-byte aligned,
four atomics where it is only 8-byte aligned (as int64 films may be).  Both must give the same
integers, with one wavelength per photon, with bundles and through planar mirrors."""
import numpy as np
import pytest

import cases
from goodphotons_b200 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hero", [1, 4])
@pytest.mark.parametrize("scene", ["cornell", "mirrors"])
@pytest.mark.parametrize("res", [1, 37])   # one pixel takes every splat; a ragged film
def test_unaligned_film_equals_aligned(gpu, scene, hero, res):
    torch = pytest.importorskip("torch")
    sc = lib.Scene(scenes.make_cornell(gpu) if scene == "cornell" else cases.make_mirrors(gpu), 0, gpu)
    cam = scenes.default_camera(gpu, res)
    words = res * res * 4
    films = []
    for shift in (0, 1):
        buf = torch.zeros(words + 2, dtype=torch.int64, device="cuda:0")
        assert buf.data_ptr() % 16 == 0
        _, en = sc.render_device(cam, 50_000, buf.data_ptr() + 8 * shift, seed_base=9, max_bounce=8, frac_bits=24,
                                 stream=torch.cuda.current_stream().cuda_stream, want_energy=True, hero_c=hero)
        film = buf.cpu().numpy()
        assert not film[:shift].any() and not film[words + shift:].any()   # nothing outside the film
        films.append((film[shift:words + shift], list(en.fx)))
    sc.close()
    assert films[0][0].reshape(-1, 4)[:, 3].sum() > 10_000
    np.testing.assert_array_equal(films[0][0], films[1][0])
    assert films[0][1] == films[1][1]
