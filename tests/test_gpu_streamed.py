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


# spp 1-3: 32 pixels a unit; 4-7: 16; from 8 on 8 pixels and 8 waves a slot on small frames
@pytest.mark.parametrize("size", [(1, 1), (7, 1), (8, 4), (9, 5), (33, 31), (31, 66)])
@pytest.mark.parametrize("spp", [1, 2, 3, 4, 7, 8, 9, 17, 64, 65])
def test_units_and_slots(size, spp):
    check(small_noise_scene(n=24, w=size[0], h=size[1], camera=synth.look_at((1.1, 0.9, 1.2))), spp, f"{size} {spp}")


# a frame wide enough that units of 16 pixels and many slots are in flight
@pytest.mark.parametrize("spp", [8, 33])
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


# thin to dense media: nearly every draw leaves its macrocell, or none does
@pytest.mark.parametrize("density", [1e-3, 0.5, 8.0, 400.0, -3.0])
@pytest.mark.parametrize("exact_log", [False, True])
def test_free_flight_over_densities(density, exact_log):
    check(small_noise_scene(n=33, w=40, h=30, density=density, exact_log=exact_log), 4, f"density {density}")


def test_emission_absorption_over_renders():
    d = small_blob_scene(n=20, w=37, h=29, emission_absorption=True, ambient=0.0)
    check(d, 9, "emission-absorption")
    check(d, 4, "emission-absorption, three renders", renders=3)
