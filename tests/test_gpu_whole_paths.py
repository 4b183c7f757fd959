"""Whole-path launches (a path traced to its end by one lane: small passes, the tail of larger
ones, renders without allocation) against the bounce-by-bounce kernels (waves).  Paths are
keyed by photon index and films are integers, so everything must be equal: the per-photon logs
of every scene kind, the films of photon counts around the limit between the two forms, and
renders whose connections overflow the queue (tested and splatted by the lane that made them)."""
import ctypes as C

import numpy as np
import pytest

import cases
from goodphotons_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture
def tuning(gpu):
    saved = gpu.get_tuning(0)
    yield lambda **kw: gpu.set_tuning(0, **kw)
    gpu.L.ftb_set_tuning(0, C.byref(saved))


@pytest.mark.parametrize("name", sorted(cases.CASES))
def test_logs_equal_bounce_by_bounce(gpu, tuning, name):
    build, res, _, mb, seed, hero = cases.CASES[name]
    sc = lib.Scene(build(gpu), 0, gpu)
    cam = scenes.default_camera(gpu, res)
    for n in (1, 33, 20_000):
        logs = []
        for regenerate in (1, 0):   # whole paths (a small streaming pass), waves
            tuning(regenerate=regenerate)
            logs.append(sc.trace_log(cam, n, seed_base=seed, max_bounce=mb, hero_c=hero))
        np.testing.assert_array_equal(logs[0], logs[1])
    sc.close()


def _device(sc, cam, n, seed, mb, hero, film, stream):
    _, en = sc.render_device(cam, n, film.data_ptr(), seed_base=seed, max_bounce=mb, frac_bits=24, stream=stream,
                             want_energy=True, hero_c=hero)
    return np.array(list(en.fx), dtype=np.int64)


@pytest.mark.parametrize("name", ["cornell", "glass", "fog_strands", "materials", "instances", "mirrors",
                                  "mirrors_fog", "glass_hero4", "mirrors_hero4"])
def test_films_equal_around_the_limit(gpu, tuning, name):
    torch = pytest.importorskip("torch")
    build, res, _, mb, seed, hero = cases.CASES[name]
    sc = lib.Scene(build(gpu), 0, gpu)
    cam = scenes.default_camera(gpu, res)
    stream = torch.cuda.current_stream().cuda_stream
    limit = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128
    for n in (limit, limit + 1, 3 * limit + 7):
        films, tallies = [], []
        for kw in (dict(regenerate=1), dict(regenerate=1, use_graphs=0), dict(regenerate=0, use_graphs=1)):
            tuning(**kw)
            film = torch.zeros((res, res, 4), dtype=torch.int64, device="cuda:0")
            tallies.append(_device(sc, cam, n, seed, mb, hero, film, stream))
            films.append(film.cpu().numpy())
        for f, t in zip(films[1:], tallies[1:]):
            np.testing.assert_array_equal(films[0], f)
            np.testing.assert_array_equal(tallies[0], t)
    sc.close()


def _bright_room(L):
    """Nearly every vertex connects and few paths die: translucent walls of albedo ~1."""
    sb = scenes.SceneBuilder()
    wall = sb.material(abi.MAT_DIFFUSE_TRANSMIT, reflect=sb.const(0.9), transmit=sb.const(0.099))
    sb.box((1.0, 1.0), (2.0, 2.0), 2.0, 0.0, wall)
    sb.area_light((0.75, 1.9, 0.75), (0.5, 0, 0), (0, 0, 0.5), (0, -1, 0), sb.blackbody(6500.0))
    return sb.build(L)


def _mirror_room(L):
    """A white room open to the camera whose back wall is a mirror: a vertex connects to the eye
    and, through the mirror, a second time."""
    sb = scenes.SceneBuilder()
    white = sb.diffuse(sb.const(0.99))
    sb.quad((0, 0, 0), (0, 0, 2), (2, 0, 0), white)
    sb.quad((0, 2, 0), (2, 0, 0), (0, 0, 2), white)
    sb.quad((0, 0, 0), (0, 2, 0), (0, 0, 2), white)
    sb.quad((2, 0, 0), (0, 0, 2), (0, 2, 0), white)
    sb.quad((0, 0, 0), (2, 0, 0), (0, 2, 0), sb.material(abi.MAT_MIRROR, reflect=sb.const(0.95)))
    sb.area_light((0.75, 1.9, 0.75), (0.5, 0, 0), (0, 0, 0.5), (0, -1, 0), sb.blackbody(6500.0))
    return sb.build(L)


def _connections(sc, cam, n, mb, hero, film, stream):
    """Connections n photons make (the occlusion rays and mirror records of a counting render)."""
    sc.set_profiling(2)
    sc.profile(True)
    _device(sc, cam, n, 3, mb, hero, film, stream)
    made = sc.profile(True).counters[3]
    sc.set_profiling(0)
    return made


@pytest.mark.parametrize("hero", [1, 4])
@pytest.mark.parametrize("room,planes", [(_bright_room, 0), (_mirror_room, 1)])
def test_connections_beyond_the_queue(gpu, tuning, room, planes, hero):
    torch = pytest.importorskip("torch")
    sc = lib.Scene(room(gpu), 0, gpu)
    cam = scenes.default_camera(gpu, 40)
    n, mb = 16_000, 24
    stream = torch.cuda.current_stream().cuda_stream
    films, tallies = [], []
    for regenerate in (1, 0):
        tuning(regenerate=regenerate)
        # a log makes the wave buffer anew, so the next render's has room for its n photons only:
        # a slot per photon and fan-out, three connection records per slot
        sc.trace_log(cam, 1)
        film = torch.zeros((40, 40, 4), dtype=torch.int64, device="cuda:0")
        tallies.append(_device(sc, cam, n, 3, mb, hero, film, stream))
        films.append(film.cpu().numpy())
    made = _connections(sc, cam, n, mb, hero, film, stream)
    assert made > 1.25 * 3 * n * (1 + planes)   # a quarter of the queue and more found it full
    if hero == 1:
        film = torch.zeros((40, 40, 4), dtype=torch.int64, device="cuda:0")
        p, info, en = abi.RenderParams(n, 3, mb, 24, 1, 0), abi.FilmInfo(), abi.Energy()
        gpu.check(gpu.L.ftb_render_forward_noalloc(sc.h, C.byref(cam), C.byref(p), C.c_void_p(film.data_ptr()),
                                                   C.byref(info), C.byref(en), C.c_void_p(stream)))
        films.append(film.cpu().numpy())
        tallies.append(np.array(list(en.fx), dtype=np.int64))
        assert made > 1.25 * 3 * abi.NOALLOC_MAX_PHOTONS   # and the fixed one of this entry point
    sc.close()
    assert films[1][..., 3].sum() > n   # (in the closed room most connections are occluded)
    for f, t in zip(films[1:], tallies[1:]):
        np.testing.assert_array_equal(films[0], f)
        np.testing.assert_array_equal(tallies[0], t)
