"""Rays at the edge of spheres (the tracer's quick miss test must never skip a sphere that is hit),
frames of every block shape and scenes without and with many spheres, bit for bit the C oracle."""
import numpy as np
import pytest
import torch

import oracle
from flyb200 import world as W
from flyb200.batch_world import BatchWorld

pytestmark = pytest.mark.gpu


def scene(spheres, rng):
    w = W.World(device="cuda")
    w.planes.append(W.Plane((0, 0, -3), (0, 0, 1), "floor"))
    w.boxes.append(W.Box((4.0, -1, -1), (4.2, 1, 1), "black"))
    for _ in range(spheres):
        r = 10.0 ** rng.uniform(-3, 0, 3) if rng.random() < 0.5 else np.full(3, 10.0 ** rng.uniform(-3, 0))
        w.spheres.append(W.Sphere(tuple(rng.uniform(-2, 2, 3)), tuple(r), "apple"))
    return w


def grazing(w, rng, per_sphere):
    """Rays whose distance from a sphere (in its own scaled space) is 1 + delta, delta from 0 over the
    rounding of the coordinates up to a percent, from origins near, far and inside."""
    o, d = [], []
    for s in w.spheres:
        c, r = np.array(s.center), np.array(s.radii)
        for _ in range(per_sphere):
            axis = rng.standard_normal(3)
            axis /= np.linalg.norm(axis)
            side = np.cross(axis, rng.standard_normal(3))
            side /= np.linalg.norm(side)
            delta = rng.choice([0.0, 1e-8, -1e-8, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5, 1e-3, -1e-2])
            back = rng.choice([0.2, 1.5, 5.0, 40.0])
            start = (c + r * (side * (1 + delta) - back * axis)).astype(np.float32)
            ray = r * axis
            o.append(start)
            d.append((ray / np.linalg.norm(ray)).astype(np.float32))
    return np.array(o, np.float32), np.array(d, np.float32)


@pytest.mark.parametrize("spheres,per_sphere", [(1, 500), (20, 400), (300, 20)])
def test_grazing_rays_match_oracle(spheres, per_sphere):
    rng = np.random.default_rng(spheres)
    w = scene(spheres, rng)
    o, d = grazing(w, rng, per_sphere)
    got = w.trace(o, d).cpu().numpy()
    ref = oracle.trace(W.pack_scene(w)[None], w._scene_shape, w.detail, origins=o[None], dirs=d[None])
    np.testing.assert_array_equal(got, ref[0])
    assert (got > 0).any()


def test_scene_without_spheres_and_far_coordinates_match_oracle():
    rng = np.random.default_rng(0)
    w = scene(0, rng)
    far = scene(5, rng)
    for s in far.spheres:
        s.center = tuple(1e5 * np.array(s.center))
    far.light_pos = (0.0, 0.0, 1e5)
    for world in (w, far):
        o = rng.uniform(-2, 2, (3000, 3)).astype(np.float32)
        d = rng.standard_normal((3000, 3))
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        got = world.trace(o, d).cpu().numpy()
        ref = oracle.trace(W.pack_scene(world)[None], world._scene_shape, world.detail, origins=o[None], dirs=d[None])
        np.testing.assert_array_equal(got, ref[0])


@pytest.mark.parametrize("batch,columns,samples", [(1, 5, 1), (1, 300, 7), (1, 400, 64), (1, 100, 65), (1, 20, 256), (3, 900, 7),
                                                   (40, 160, 7)])
def test_block_shapes_of_the_eye_match_oracle(batch, columns, samples):
    rng = np.random.default_rng(columns)
    az, el = rng.uniform(-np.pi, np.pi, (columns, samples)), rng.uniform(-1.2, 1.2, (columns, samples))
    dirs = np.stack([np.cos(el) * np.cos(az), np.cos(el) * np.sin(az), np.sin(el)], -1)
    weights = rng.random(samples)
    b = BatchWorld([W.make_room(i)[0] for i in range(batch)], device="cuda")
    b.set_eye(dirs, weights)
    eye = np.c_[rng.uniform(-1.5, 1.5, (batch, 2)), rng.uniform(0.8, 1.5, batch)]
    heading = rng.uniform(-np.pi, np.pi, batch)
    forward = np.c_[np.cos(heading), np.sin(heading), np.zeros(batch)]
    left = np.c_[-np.sin(heading), np.cos(heading), np.zeros(batch)]
    up = np.cross(forward, left)
    got = b.column_radiance(eye, forward, left, up).cpu().numpy()
    ref = oracle.trace(np.stack([W.pack_scene(s) for s in b.worlds]), b._scene_shape, b.detail, origins=eye,
                       eye_dirs=dirs.reshape(-1, 3), pose=np.concatenate([forward, left, up], 1), weights=weights,
                       shared_origin=True, batch=batch)
    np.testing.assert_array_equal(got, ref)
