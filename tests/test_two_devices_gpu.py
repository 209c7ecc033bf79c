"""Row kernels and the reverse scan in one process on two devices: what a launch needs is allowed on each of them."""
import ctypes

import pytest
import torch

from warpstate_ai_b200.ops import _ext


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="two devices")
def test_norm_backward_and_reverse_scan_on_a_second_device():
    _ext.require()
    results = []
    for device in ("cuda:0", "cuda:1"):
        with torch.cuda.device(device):
            r = lambda *s: torch.linspace(-1, 1, torch.Size(s).numel(), device=device).view(s)  # noqa: E731
            dx, _, dw = torch.ops.ws_b200.rmsnorm_bwd(r(700, 256).bfloat16(), r(700, 256), r(700) + 2, r(256), None, None, False)
            g, w, logits = r(1, 3, 2, 4096), r(1, 3, 2, 4096), r(3, 2)
            out, partials = torch.empty_like(g).bfloat16(), torch.empty(32, 3, device=device)
            p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
            assert _ext.cdll().ws_memory_scan_bwd(p(g), p(w), p(logits[0]), p(logits[1]), p(logits[2]), p(out), p(partials), 1, 3, 2,
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            results.append([t.cpu() for t in (dx, dw, out, partials)])
    assert all(torch.equal(a, b) for a, b in zip(*results))
