"""The streamed render loop of plain jobs at the sizes where its bookkeeping
can go wrong -- pixels per unit, waves per slot, the last chunk of a frame, a
ring that wraps -- and its two shortcuts, pixels whose rays cannot meet the
volume and free-flight draws that leave their macrocell: frames and work
counters equal the oracle's, bit for bit."""
import numpy as np
import pytest

import oracle
from barney_b200 import synth
from tests.helpers import assert_bitexact, gpu_render, small_blob_scene, small_noise_scene

pytestmark = pytest.mark.gpu


def check(d, spp, what, renders=1):
    img, st = gpu_render(d, spp, renders=renders)
    acc = np.zeros((d["height"], d["width"], 4), np.float32)
    comp = np.zeros_like(acc) if d.get("compensated_accum") else None
    _, _, ost = oracle.render(oracle.Scene(d), 0, spp * renders, accum=acc, comp=comp)
    assert_bitexact(img, oracle.resolve(acc, spp * renders, comp=comp), what)
    if renders == 1:
        assert (st["samples"], st["mc_visits"], st["rays"]) == (ost["samples"], ost["mc_visits"], ost["rays"])
    assert st["error_flags"] == 0


# small frames: 32 pixels a unit at 1 spp, 16 at 2-3, 8 from 4 on (8 waves a slot from 8 on)
@pytest.mark.parametrize("size", [(1, 1), (7, 1), (8, 4), (9, 5), (33, 31), (31, 66)])
@pytest.mark.parametrize("spp", [1, 2, 3, 4, 7, 8, 9, 17, 64, 65])
def test_units_and_slots(size, spp):
    check(small_noise_scene(n=24, w=size[0], h=size[1], camera=synth.look_at((1.1, 0.9, 1.2))), spp, f"{size} {spp}")


# a frame wide enough that units of 32 (2 spp) and 16 pixels and many slots are in flight
@pytest.mark.parametrize("spp", [2, 5, 8, 33])
def test_wide_frame(spp):
    check(small_blob_scene(n=20, w=1021, h=563), spp, f"wide {spp}")


# what a pixel outside the volume adds: black with alpha 1 (one addition),
# colours, alpha that rounds, a gradient per row, colours above the clamp, NaN
# (the clamp's value)
@pytest.mark.parametrize("bg", [(0.0, 0.0, 0.0, 1.0), (0.2, 0.0, 0.7, 1.0), (0.0, 0.0, 0.0, 0.3), (0.1, 0.2, 0.3, -1.0),
                                (25.0, 0.0, 3.0, 1.0), (-0.5, 0.0, -0.0, 0.0), (np.nan, 0.0, -1.0, 1.0),
                                (0.0, -np.inf, np.nan, 1.0)])
@pytest.mark.parametrize("comp", [False, True])
def test_pixels_outside_the_volume(bg, comp):
    d = small_noise_scene(n=20, w=70, h=41, bg_color=bg, compensated_accum=comp, majorant_round_up=comp,
                          camera=synth.look_at((4.0, 3.0, 4.0)))
    check(d, 5, f"bg {bg}")
    check(d, 3, f"bg {bg}, three renders", renders=3)


# cameras near, far, beside, inside, grazing; narrow and wide fields of view
@pytest.mark.parametrize("seed", range(40))
def test_culled_pixels_over_cameras(seed):
    rng = np.random.default_rng(seed)
    r = float(np.exp(rng.uniform(np.log(0.3), np.log(50.0))))
    v = rng.normal(size=3)
    pos = 0.5 + r * v / np.linalg.norm(v)
    fovy = float(np.exp(rng.uniform(np.log(0.05 if seed % 4 == 0 else 5.0), np.log(140.0))))
    target = rng.uniform(-0.3, 1.3, size=3) if seed % 2 else (0.5, 0.5, 0.5)
    up = tuple(rng.normal(size=3)) if seed % 3 else (0.0, 1.0, 0.0)
    cam = synth.look_at(pos, target=target, fovy=fovy, up=up)
    vox = synth.blobs(17, seed)[:, :13, :9].copy() if seed % 5 == 0 else synth.blobs(17, seed)
    d = synth.scene(vox, "f32", 61, 37, synth.tf_linear_ramp(64), 20.0, cam, ambient=1.0)
    if seed % 5 == 0:
        d["origin"] = (0.3, -0.2, 0.1)
    if seed % 7 == 0:
        d["cut_plane"] = (0.0, 1.0, 0.0, -0.5)
    check(d, 2, f"camera {seed}")


# cameras close to the volume, in it, on the planes of its faces and turned away from
# it: corners beside and behind the camera; cut planes through, before and beyond it
@pytest.mark.parametrize("seed", range(60))
def test_culled_pixels_beside_the_volume(seed):
    rng = np.random.default_rng(1000 + seed)
    pos = rng.uniform(-0.7, 1.7, size=3)
    if seed % 4 == 1:
        pos[seed % 3] = float(seed % 8 > 4)
    if seed % 4 == 2:
        pos[seed % 3] = (-1e-3, 1.001, -0.02, 1.3)[seed // 4 % 4]
    target = pos + rng.normal(size=3) if seed % 3 else np.array((0.5, 0.5, 0.5)) + 2 * (pos - 0.5)
    cam = synth.look_at(pos, target=target, fovy=float(rng.uniform(20.0, 170.0)), up=tuple(rng.normal(size=3)))
    d = synth.scene(synth.blobs(17, seed), "f32", 61, 37, synth.tf_linear_ramp(64), 20.0, cam, ambient=1.0,
                    bg_color=(0.1, 0.0, 0.2, 1.0))
    if seed % 5 == 3:
        n = rng.normal(size=3)
        d["cut_plane"] = (*(float(x) for x in n), float(rng.choice([-6.0, -0.5, 0.2, 6.0])))
    check(d, 2, f"camera {seed}")


# thin to dense media: nearly every draw leaves its macrocell, or none does
@pytest.mark.parametrize("density", [1e-3, 0.5, 8.0, 400.0, -3.0])
@pytest.mark.parametrize("exact_log", [False, True])
def test_free_flight_over_densities(density, exact_log):
    check(small_noise_scene(n=33, w=40, h=30, density=density, exact_log=exact_log), 4, f"density {density}")


def test_emission_absorption_over_renders():
    d = small_blob_scene(n=20, w=37, h=29, emission_absorption=True, ambient=0.0)
    check(d, 9, "emission-absorption")
    check(d, 4, "emission-absorption, three renders", renders=3)


# Batches: lanes of a warp hold paths of several jobs.  The jobs differ in storage,
# size, sums, background and camera; some see nothing of their volume.
def batch_scenes(n):
    out = []
    for i in range(n):
        kw = {"camera": synth.look_at((4.0, 3.0, 4.0) if i % 7 == 5 else (1.1, 0.9, 1.2) if i % 3 else (2.0, 1.5, 2.0),
                                      target=(9.0, 9.0, 9.0) if i % 7 == 3 else synth.CUBE_CENTRE)}
        if i % 4 == 1:
            kw.update(compensated_accum=True, majorant_round_up=True)
        if i % 5 == 2:
            kw["bg_color"] = (0.2, 0.0, 0.7, 1.0)
        w, h = [(33, 31), (7, 1), (9, 5), (31, 66), (64, 24)][i % 5]
        out.append(small_noise_scene(n=[24, 13, 20][i % 3], w=w, h=h, dtype=["f32", "u8", "f16"][i % 3], **kw))
    return out


def check_batch(scenes, spps, graphs, renders):
    import barney_b200 as bn
    ctx = bn.Context()
    ctx.set_graphs(graphs)
    rs = [bn.VolumeRenderer(d, context=ctx) for d in scenes]
    for r, spp in zip(rs, spps):
        r.set_spp(spp)
    for _ in range(renders):
        ctx.render_batch(rs)
    assert ctx.stats()["error_flags"] == 0
    for i, (r, d, spp) in enumerate(zip(rs, scenes, spps)):
        acc = np.zeros((d["height"], d["width"], 4), np.float32)
        comp = np.zeros_like(acc) if d.get("compensated_accum") else None
        oracle.render(oracle.Scene(d), 0, spp * renders, accum=acc, comp=comp)
        assert_bitexact(r.read(), oracle.resolve(acc, spp * renders, comp=comp), f"job {i}, {spp} spp")
        r.close()
    ctx.close()


# at most 4 jobs without graphs travel as a kernel parameter
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("n", [2, 4, 5, 12])
@pytest.mark.parametrize("spps", [[1], [2], [4], [9], [1, 7, 8, 33, 65]])
def test_batches(n, spps, graphs):
    check_batch(batch_scenes(n), [spps[i % len(spps)] for i in range(n)], graphs, 2)


# 31 jobs as a parameter and 32 as a table: a large frame beside its volume carries the
# paths that make the parameter the choice
@pytest.mark.parametrize("n", [31, 32])
def test_batches_at_the_parameter_limit(n):
    scenes = batch_scenes(n - 1)
    scenes.insert(3, small_noise_scene(n=12, w=1024, h=1024, camera=synth.look_at((2.0, 1.5, 2.0), target=(9.0, 9.0, 9.0))))
    spps = [[1, 7, 8, 33][i % 4] for i in range(n - 1)]
    spps.insert(3, 42)
    check_batch(scenes, spps, False, 1)


# enough chunks for units of 16 pixels at 8 spp, and of 32 below
@pytest.mark.parametrize("spp", [2, 4, 9])
def test_large_batch(spp):
    scenes = [small_noise_scene(n=20, w=509, h=601, camera=synth.look_at(p))
              for p in ((4.0, 3.0, 4.0), (6.0, -3.0, 2.0), (3.0, 9.0, 4.0))]
    check_batch(scenes, [spp] * 3, False, 1)
