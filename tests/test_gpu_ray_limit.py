"""The number of rays a call takes: refused, before anything is launched or read, where 32-bit counters
would wrap."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

SFTG_RAY_MAX, SFTG_E_LIMIT = 0xFFF00000, -4


@pytest.mark.parametrize("n", [SFTG_RAY_MAX + 1, 0xFFFFFFFF])
@pytest.mark.parametrize("call", ["sftg_raycast", "sftg_raycast_device"])
def test_too_many_rays(renderer, call, n):
    ctx, buf = renderer.lib.sft_get_gpu_context(), torch.zeros(256, dtype=torch.uint8, device="cuda")
    assert getattr(renderer.lib, call)(ctx, C.c_void_p(buf.data_ptr()), n, C.c_void_p(buf.data_ptr() + 128)) == SFTG_E_LIMIT
    assert b"rays" in renderer.lib.sftg_last_error(ctx)
    torch.cuda.synchronize()
