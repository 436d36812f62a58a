"""Freed device blocks are kept for the next allocation of their size: volumes
opened one after another in reused memory render as in fresh memory, an
injected allocation failure is not hidden by a kept block, the last context's
end gives the memory back, and a release disturbs no stream capture."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from barney_b200 import synth
from tests.helpers import assert_bitexact, oracle_render, small_noise_scene

pytestmark = pytest.mark.gpu


def test_reopened_volumes():
    import barney_b200 as bn
    ctx = bn.Context()
    try:
        for seed in (0, 1, 2, 0):
            vol = synth.value_noise(40, seed)
            d = synth.config2(vol=vol, width=40, height=28)
            d["compensated_accum"] = seed == 1
            r = bn.VolumeRenderer(d, context=ctx)
            r.set_spp(2)
            r.render()
            ref, _, _ = oracle_render(dict(d, compensated_accum=False), 2)
            got = r.read()
            r.close()
            if seed == 1:  # two waves: the compensated sum differs by its last rounding at most
                assert np.allclose(got, ref, rtol=2e-7, atol=0)
            else:
                assert_bitexact(got, ref, f"seed {seed}")
        vox = np.ascontiguousarray(synth.value_noise(40, 3))
        L = ctx.L
        L.bnxInjectAllocationFailure(0)
        assert not L.bnTextureData3DCreate(ctx.ctx, 0, bn.BN_FLOAT32, 40, 40, 40, vox.ctypes.data)
        assert L.bnGetLastError() == 6
        L.bnClearLastError()
    finally:
        L.bnxInjectAllocationFailure(-1)
        ctx.close()


def test_memory_goes_back_with_the_last_context():
    code = """
import torch, barney_b200 as bn
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
vox = torch.zeros((256, 512, 512), device="cuda"); torch.cuda.synchronize()
ctx = bn.Context(); before = free()
for _ in range(3):
    t = ctx.L.bnTextureData3DCreate(ctx.ctx, 0, bn.BN_FLOAT32, 512, 512, 256, vox.data_ptr()); bn.check()
    ctx.L.bnRelease(t); bn.check()
assert before - free() <= (256 << 20) + (64 << 20), "one block is held, not three"
ctx.close()
assert free() >= before, "nothing is held without a context"
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


def test_memory_goes_back_on_request_and_after_the_last_context():
    code = """
import torch, barney_b200 as bn
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
vox = torch.zeros((256, 512, 512), device="cuda"); torch.cuda.synchronize()
MB = 1 << 20
ctx = bn.Context()
def cycle():
    t = ctx.L.bnTextureData3DCreate(ctx.ctx, 0, bn.BN_FLOAT32, 512, 512, 256, vox.data_ptr()); bn.check()
    ctx.L.bnRelease(t); bn.check()
cycle(); ctx.set_memory_cache(0); before = free()
cycle()
assert before - free() <= 8 * MB, "with no cache a release is given back at once"
ctx.set_memory_cache(300 * MB)
cycle()
assert before - free() >= 256 * MB, "kept"
other = bn.Context(); other.set_memory_cache(0); other.close()
assert before - free() <= 8 * MB, "trimmed"
cycle(); cycle()
s = bn.Server(ctx, max_slots=2, slice_waves=1); s.reserve(512 * MB)
ctx.close()
s.close()
assert free() >= before - 8 * MB, "the server's buffers, released after the last context"
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


def test_path_rings_come_with_the_first_plain_frame():
    code = """
import torch, barney_b200 as bn
from barney_b200 import synth
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
MB = 1 << 20
d = synth.config2(vol=synth.value_noise(16, 0), width=24, height=16)
keep = bn.Context()
for bounces in (0, 2):  # the kernels' code is loaded on their first launch
    r = bn.VolumeRenderer(dict(d, max_volume_bounces=bounces), context=keep); r.render(); r.close()
before = free()
ctxs = [bn.Context() for _ in range(4)]
assert before - free() <= 8 * MB, "contexts alone"
rs = [bn.VolumeRenderer(dict(d, max_volume_bounces=2), context=c) for c in ctxs]
for r in rs: r.render()
assert before - free() <= 32 * MB, "multi-scatter frames need no rings"
r = bn.VolumeRenderer(d, context=ctxs[0]); r.render()
assert 64 * MB <= before - free() <= 112 * MB, "one context's rings"
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


def test_failed_allocations_of_a_context():
    """A context that cannot be created leaves nothing behind, and one whose
    path rings find no memory renders the same frames with smaller ones."""
    import barney_b200 as bn
    L = bn.lib()
    d = small_noise_scene(n=20, w=301, h=203)
    try:
        L.bnxInjectAllocationFailure(0)
        assert not L.bnContextCreate(1, None, 0, None)
        assert L.bnGetLastError() == 6
        L.bnClearLastError()
        for batch in (False, True):
            ctx = bn.Context()
            rs = [bn.VolumeRenderer(d, context=ctx) for _ in range(2)]
            for r in rs:
                r.set_spp(9)
            if batch:
                L.bnxInjectAllocationFailure(2)  # the batch's job and chunk tables, then the rings
                ctx.render_batch(rs)
            else:
                L.bnxInjectAllocationFailure(0)
                rs[0].render()
            bn.check()
            assert_bitexact(rs[0].read(), oracle_render(d, 9)[0], f"smaller rings, batch {batch}")
            # the injected failure was the rings': none is left for this one
            t = L.bnTextureData3DCreate(ctx.ctx, 0, bn.BN_FLOAT32, 2, 2, 2, np.zeros(8, np.float32).ctypes.data)
            bn.check()
            L.bnRelease(t)
            for r in rs:
                r.close()
            ctx.close()
    finally:
        L.bnxInjectAllocationFailure(-1)


def test_release_during_an_applications_capture():
    import torch
    import barney_b200 as bn
    ctx = bn.Context()
    d = small_noise_scene(n=16, w=24, h=16)
    r = bn.VolumeRenderer(d, context=ctx)
    r.render()
    x = torch.zeros(64, device="cuda")
    s, g, errors = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []

    def work():
        try:
            r.resize(40, 30)
            r.close()
            r2 = bn.VolumeRenderer(d, context=ctx)
            r2.render()
            r2.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        x.add_(1)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x.add_(1)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    ctx.close()
    assert not errors
    assert (x == 2).all()


def test_release_while_another_context_captures():
    import barney_b200 as bn
    scenes = [small_noise_scene(n=16, w=24, h=16 + i) for i in range(6)]
    a, b = bn.Context(), bn.Context()
    rs = [bn.VolumeRenderer(d, context=a) for d in scenes]
    for r in rs:
        r.set_spp(2)
    stop, errors = threading.Event(), []

    def opens():
        try:
            while not stop.is_set():
                bn.VolumeRenderer(scenes[0], context=b).close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    t = threading.Thread(target=opens)
    t.start()
    try:
        for i in range(200):  # another batch shape every time: a capture each
            n = 1 + i % 6
            for r in rs[:n]:
                r.accum_reset()
            a.render_batch(rs[:n])
    finally:
        stop.set()
        t.join()
    assert not errors
    for r, d in zip(rs, scenes):
        assert_bitexact(r.read(), oracle_render(d, 2)[0], "batch beside releases")
        r.close()
    b.close()
    a.close()


def test_blocks_an_application_may_still_use_go_back_to_cuda():
    """A colour pointer handed out, and work on an application's stream: the
    release waits for them and the next allocation does not reuse the block."""
    import torch
    import barney_b200 as bn
    d = small_noise_scene(n=16, w=256, h=256)
    ctx = bn.Context()
    r = bn.VolumeRenderer(d, context=ctx)
    r.render()
    ref = r.read()
    ptr = ctx.L.bnxFrameBufferDevicePointer(r.fb)
    dst = torch.zeros((256, 256, 4), device="cuda")
    libcudart = _cudart()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)  # some 50 ms before the application's copy
        assert libcudart.cudaMemcpyAsync(dst.data_ptr(), ptr, dst.numel() * 4, 3, s.cuda_stream) == 0
    r.close()
    r = bn.VolumeRenderer(dict(d, bg_color=(1.0, 0.5, 0.25, 1.0)), context=ctx)
    r.render()
    torch.cuda.synchronize()
    assert_bitexact(dst.cpu().numpy(), ref, "the application's copy")
    r.close()
    ctx.close()


def _cudart():
    import ctypes
    import torch  # noqa: F401
    path = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)
    lib = ctypes.CDLL(path)
    lib.cudaMemcpyAsync.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_void_p]
    return lib
