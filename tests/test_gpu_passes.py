"""Passes and their buffers: a render that is one streaming pass takes the room of both wave
buffers, one of several passes alternates between two.  Small buffers (the tuning's wave_slots)
make the refill, the second buffer and the direction-ordered queues of large scenes run at
small photon counts; every film and tally must equal the same photons traced in whole-path
launches."""
import ctypes as C

import numpy as np
import pytest

import cases
from goodphotons_b200 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture
def tuning(gpu):
    saved = gpu.get_tuning(0)
    yield lambda **kw: gpu.set_tuning(0, **kw)
    gpu.L.ftb_set_tuning(0, C.byref(saved))


def _solo(gpu, torch, sc, cam, n, seed, mb, hero):
    """n photons in renders of at most 50,000 (whole-path launches)."""
    film = torch.zeros((cam.res_y, cam.res_x, 4), dtype=torch.int64, device="cuda:0")
    fx = np.zeros(5, dtype=np.int64)
    for first in range(0, n, 50_000):
        _, en = sc.render_device(cam, min(50_000, n - first), film.data_ptr(), seed_base=seed + first, max_bounce=mb,
                                 frac_bits=24, stream=torch.cuda.current_stream().cuda_stream, want_energy=True,
                                 hero_c=hero)
        fx += np.array(list(en.fx), dtype=np.int64)
    return film.cpu().numpy(), fx


@pytest.mark.parametrize("slots", [1 << 12, (1 << 14) + 1, 1 << 22])
@pytest.mark.parametrize("heroes", [(1, 1, 1), (1, 4, 1, 4)])   # one pass; a pass per class change
def test_passes_equal_whole_paths(gpu, tuning, slots, heroes):
    torch = pytest.importorskip("torch")
    scs = [lib.Scene(scenes.make_cornell(gpu), 0, gpu), lib.Scene(scenes.make_glass(gpu, level=3), 0, gpu)]
    cam = scenes.default_camera(gpu, 24)
    jobs, films = [], []
    for k, hero in enumerate(heroes):
        film = torch.zeros((24, 24, 4), dtype=torch.int64, device="cuda:0")
        films.append(film)
        jobs.append(dict(scene=scs[k % 2], cam=cam, d_film=film.data_ptr(), n=90_001 + 13 * k, seed_base=1000 * k,
                         max_bounce=8 + 4 * (k % 2), frac_bits=24, hero_c=hero))
    stream = torch.cuda.current_stream().cuda_stream
    tuning(wave_slots=slots)
    _, ens = gpu.render_batch(jobs, stream=stream)
    tuning(wave_slots=1 << 22)
    for job, film, en in zip(jobs, films, ens):
        ref, fx = _solo(gpu, torch, job["scene"], cam, job["n"], job["seed_base"], job["max_bounce"], job["hero_c"])
        np.testing.assert_array_equal(film.cpu().numpy(), ref)
        np.testing.assert_array_equal(np.array(list(en.fx), dtype=np.int64), fx)
    for sc in scs:
        sc.close()


@pytest.mark.parametrize("name,build", [
    ("glass", lambda L: scenes.make_glass(L, freq=90)),                # ~18 k nodes
    ("fog_strands", lambda L: scenes.make_fog_strands(L, n_strands=40_000)),
    ("instanced", lambda L: scenes.make_glass_instanced(L, level=6)),   # the large hierarchy is the BLAS's
])
def test_ordered_queues_of_large_scenes(gpu, tuning, name, build):
    torch = pytest.importorskip("torch")
    sc = lib.Scene(build(gpu), 0, gpu)
    cam = scenes.default_camera(gpu, 40)
    n, mb = 150_000, 12
    ref, fx = _solo(gpu, torch, sc, cam, n, 5, mb, 1)
    for kw in (dict(wave_slots=30_000, sort_rays=1), dict(wave_slots=30_000, sort_rays=1, regenerate=0)):
        tuning(**kw)
        film = torch.zeros((40, 40, 4), dtype=torch.int64, device="cuda:0")
        _, en = sc.render_device(cam, n, film.data_ptr(), seed_base=5, max_bounce=mb, frac_bits=24,
                                 stream=torch.cuda.current_stream().cuda_stream, want_energy=True)
        np.testing.assert_array_equal(film.cpu().numpy(), ref)
        np.testing.assert_array_equal(np.array(list(en.fx), dtype=np.int64), fx)
    sc.close()


@pytest.mark.parametrize("n_jobs", [3, 40, 64, 65, 128, 129])   # tally tables of 64, 128 and 256 rows
def test_ordered_queues_of_mixed_scenes(gpu, tuning, n_jobs):
    """Each path is put on the grid of its own job's scene, and tallied to its own job."""
    torch = pytest.importorskip("torch")
    scs = [lib.Scene(scenes.make_cornell(gpu), 0, gpu), lib.Scene(scenes.make_glass(gpu, freq=90), 0, gpu),
           lib.Scene(scenes.make_fog_strands(gpu, n_strands=40_000), 0, gpu)]
    cam = scenes.default_camera(gpu, 20)
    jobs, films = [], []
    for k in range(n_jobs):
        film = torch.zeros((20, 20, 4), dtype=torch.int64, device="cuda:0")
        films.append(film)
        jobs.append(dict(scene=scs[k % 3], cam=cam, d_film=film.data_ptr(), n=120_000 // n_jobs + k,
                         seed_base=10_000 * k, max_bounce=6 + k % 5, frac_bits=24))
    tuning(wave_slots=20_000, sort_rays=1)
    _, ens = gpu.render_batch(jobs, stream=torch.cuda.current_stream().cuda_stream)
    tuning(wave_slots=1 << 22)
    for job, film, en in zip(jobs, films, ens):
        ref, fx = _solo(gpu, torch, job["scene"], cam, job["n"], job["seed_base"], job["max_bounce"], 1)
        np.testing.assert_array_equal(film.cpu().numpy(), ref)
        np.testing.assert_array_equal(np.array(list(en.fx), dtype=np.int64), fx)
    for sc in scs:
        sc.close()
