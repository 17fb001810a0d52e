"""Copies between pageable arrays and the device through several threads' page-locked slots:
sizes around the staging limit and its chunks give the bytes that small direct copies give,
also from several Python threads with handles of their own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def renderer(rg):
    r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=8, resolutionHeight=8, samples=1))
    r.set_scene(rg.Scene.builtin(1, 1))
    return r


def rays_of(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[:, 2] = -np.abs(d[:, 2]) - 0.5
    return np.concatenate([rng.uniform(-2, 2, (n, 3)).astype(np.float32), d], axis=1)


def in_pieces(r, rays, step=5000):
    parts = [r.trace_closest(rays[k:k + step]) for k in range(0, len(rays), step)]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


# 24 bytes a ray in, 12 and 4 out: one ray; the small-batch limit (16384); the limit of a warp per
# ray (32768; the pieces compared with are below it); around 3 MB in (131072) and 3 MB of t, u, v
# (262144) with and without a ragged chunk; several chunks a worker
@pytest.mark.parametrize("n", [1, 16384, 16385, 32768, 32769, 131071, 131072, 131073, 262144, 700001])
def test_query_sizes(rg, n):
    r = renderer(rg)
    rays = rays_of(n, n)
    tuv, prim = r.trace_closest(rays)
    want_tuv, want_prim = in_pieces(r, rays)
    np.testing.assert_array_equal(prim, want_prim)
    np.testing.assert_array_equal(tuv, want_tuv)
    occ = r.trace_any(rays, np.full(n, 4.0, np.float32))
    want = np.concatenate([r.trace_any(rays[k:k + 5000], np.full(len(rays[k:k + 5000]), 4.0, np.float32))
                           for k in range(0, n, 5000)])
    np.testing.assert_array_equal(occ, want)
    r.close()


def test_sizes_once_slots_are_there(rg):
    """The first large batch makes the slots; around 3 MB in, with and without ragged chunks."""
    r = renderer(rg)
    r.trace_closest(rays_of(1500000, 1))
    for n in (131071, 131072, 131073, 174763, 400001):
        rays = rays_of(n, n)
        want_tuv, want_prim = in_pieces(r, rays)
        tuv, prim = r.trace_closest(rays)
        np.testing.assert_array_equal(prim, want_prim)
        np.testing.assert_array_equal(tuv, want_tuv)
    r.close()


def test_threads_with_their_own_handles(rg):
    errors = []

    def work(k):
        try:
            r = renderer(rg)
            rays = rays_of(200000 + 1111 * k, k)
            want = in_pieces(r, rays)
            for _ in range(3):
                got = r.trace_closest(rays)
                np.testing.assert_array_equal(got[0], want[0])
                np.testing.assert_array_equal(got[1], want[1])
            r.close()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
