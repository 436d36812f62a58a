"""The bounds-checked build (libbarney_b200_bc.so, -DBNB_BOUNDS_CHECK): every
indexed access of the render and macrocell kernels is checked against its
array; on small and ragged volumes of every storage type, with isosurfaces,
multi-scatter paths, batches and accumulation, it counts no out-of-range
access and renders exactly the oracle's frames.  It runs in a child process,
since a process loads one build of the library."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import numpy as np
import oracle
import barney_b200 as bn
from barney_b200 import synth
from tests.helpers import assert_bitexact, oracle_render, small_blob_scene, small_noise_scene

scenes = [
    small_noise_scene(n=8, w=19, h=13),
    small_noise_scene(n=13, w=23, h=17, dtype="u8", phase="simple"),
    small_noise_scene(n=21, w=16, h=16, dtype="f16", max_volume_bounces=3, anisotropy=0.5),
    small_noise_scene(n=32, w=24, h=20, dtype="u16", iso={"value": 0.5, "opacity": 0.8}),
    small_noise_scene(n=17, w=21, h=15, dtype="bf16", cut_plane=(0.0, 1.0, 0.0, -0.4)),
    small_blob_scene(n=9, w=17, h=11, volume=False, iso={"value": 0.2}),
    small_blob_scene(n=24, w=31, h=7, compensated_accum=False, principled={"enabled": 1}, phase="hg",
                     max_volume_bounces=2),
]
ragged = synth.value_noise(21, 3)[:, 2:15, 4:13].copy()
scenes.append(dict(synth.config2(vol=ragged, width=15, height=11), spacing=(1 / 8, 1 / 12, 1 / 20)))
# rows read as vectors: a warp of macrocells, one that ends inside it, and more
for shape, dtype in (((10, 9, 264), "f32"), ((9, 17, 248), "u8"), ((3, 12, 520), "f16"), ((12, 3, 8), "u16")):
    vol = synth.to_storage(np.random.default_rng(1).random(shape).astype(np.float32), dtype)
    scenes.append(synth.scene(vol, dtype, 18, 13, synth.tf_linear_ramp(64), 20.0, synth.DEFAULT_CAMERA))
ctx = bn.Context()
assert ctx.L.bnxBoundsViolations(ctx.ctx) == 0, "bounds-checked build expected"
for i, d in enumerate(scenes):
    r = bn.VolumeRenderer(d, color_format="float4", context=ctx)
    r.set_spp(3)
    r.render()
    r.render()  # a second launch accumulates (reads the accumulation buffer)
    ref, _, _ = oracle_render(d, 6)
    assert_bitexact(r.read(), ref, f"scene {i}")
    r.close()
# the streamed loop's rings: several slots a unit, rings that wrap, units of 32, 16 and 8 pixels
near = dict(camera=synth.look_at((1.1, 0.9, 1.2)))
for d, spp in ((small_noise_scene(n=20, w=70, h=61, **near), 1), (small_noise_scene(n=20, w=70, h=61, **near), 2),
               (small_noise_scene(n=20, w=70, h=61, **near), 65), (small_noise_scene(n=20, w=33, h=31, **near), 33),
               (small_noise_scene(n=20, w=401, h=205, density=5.0, **near), 8), (small_blob_scene(n=20, w=1021, h=563), 8),
               (small_blob_scene(n=20, w=61, h=43, emission_absorption=True, ambient=0.0), 19),
               (small_noise_scene(n=20, w=61, h=43, compensated_accum=True, majorant_round_up=True), 17)):
    r = bn.VolumeRenderer(d, color_format="float4", context=ctx)
    r.set_spp(spp)
    r.render()
    acc = np.zeros((d["height"], d["width"], 4), np.float32)
    comp = np.zeros_like(acc) if d.get("compensated_accum") else None
    oracle.render(oracle.Scene(d), 0, spp, accum=acc, comp=comp)
    assert_bitexact(r.read(), oracle.resolve(acc, spp, comp=comp), f"{d['width']}x{d['height']} {spp} spp")
    r.close()
plain = [small_noise_scene(n=[16, 20, 13][i % 3], w=40 + 23 * i, h=61 - 3 * i, dtype=["f32", "u8", "f16"][i % 3], **near)
         for i in range(9)]
for graphs in (False, True):
    for n in (3, 9):  # a kernel parameter, a table
        ctx.set_graphs(graphs)
        rs = [bn.VolumeRenderer(d, color_format="float4", context=ctx) for d in plain[:n]]
        for i, r in enumerate(rs):
            r.set_spp([1, 9, 33][i % 3])
        ctx.render_batch(rs)
        for i, (r, d) in enumerate(zip(rs, plain)):
            assert_bitexact(r.read(), oracle_render(d, [1, 9, 33][i % 3])[0], f"job {i}")
            r.close()
rs = [bn.VolumeRenderer(d, color_format="float4", context=ctx) for d in scenes[:4]]
for r in rs:
    r.set_spp(2)
ctx.render_batch(rs)
for r, d in zip(rs, scenes[:4]):
    ref, _, _ = oracle_render(d, 2)
    assert_bitexact(r.read(), ref, "batch")
    r.close()
n = ctx.L.bnxBoundsViolations(ctx.ctx)
ctx.close()
assert n == 0, f"{n} out-of-range accesses"
print("bounds-checked build: 0 out-of-range accesses")
"""


def test_bounds_checked_build_counts_no_out_of_range_access():
    from barney_b200 import build as _build
    lib = _build.build(bounds_check=True)
    env = dict(os.environ, BARNEY_B200_LIBRARY=lib, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "0 out-of-range accesses" in r.stdout
