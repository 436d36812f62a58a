"""Freed device blocks are kept for the next allocation of their size: volumes
opened one after another in reused memory render as in fresh memory, an
injected allocation failure is not hidden by a kept block, and the last
context's end gives the memory back."""
import os
import subprocess
import sys

import numpy as np
import pytest

from barney_b200 import synth
from tests.helpers import assert_bitexact, oracle_render

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
