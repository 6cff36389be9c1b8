"""The bounds-checked debug build checks the indices of every convolution path: gathers of odd and
even channel counts, element by element, and the weight gradient on the image.  In a child process
because the build variant is chosen when the library loads."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import sys, torch
sys.path.insert(0, %r)
from necklace_b200 import _lib
from necklace_b200.ops import check_status
from necklace_b200.ops import conv as cv
torch.manual_seed(0)

def seen(fn, tu):
    fn()
    torch.cuda.synchronize()
    check_status()
    assert tu in _lib.debug_bounds_seen(), (tu, "no check was evaluated")
    assert _lib.debug_bounds() == {}
    _lib.debug_bounds_seen()

x = lambda *s: torch.randn(*s, device="cuda").bfloat16()
_lib.debug_bounds_seen()
seen(lambda: cv.im2col(x(2, 20, 20, 3), 7, 7, 2, 3), "conv")          # rows in shared memory
seen(lambda: cv.im2col(x(2, 9, 9, 16), 3, 3, 3, 1), "conv")           # 16 bytes at a time
seen(lambda: cv.im2col(x(1, 2, 2, 4099), 3, 3, 1, 1), "conv")         # element by element
seen(lambda: cv.col2im(x(2 * 9 * 9, 144), (2, 9, 9, 16), 3, 3, 1, 1), "conv")
for (N, H, W, ci, co, k, s) in [(2, 9, 9, 16, 24, 3, 1), (1, 11, 7, 8, 136, 3, 2), (5, 7, 7, 72, 264, 1, 2)]:
    img, w = x(N, H, W, ci), x(co, k * k * ci)
    y = cv._conv_fwd(img, w, k, k, s, k // 2)
    cv._conv_dgrad(y.reshape(-1, co), w, img.shape, k, k, s, k // 2)
    seen(lambda: cv._conv_wgrad(img, y.reshape(-1, co), w, k, k, s, k // 2, None, False), "convimg")
for (ci, co, s) in [(16, 12, 1), (16, 24, 3), (4099, 8, 1)]:          # gathered layers, there and back
    conv = cv.Conv2d(ci, co, 3, s, 1, device="cuda")
    seen(lambda: conv(x(1, 4, 4, ci).requires_grad_(True)).float().sum().backward(), "conv")
print("CONV_BOUNDS_OK")
'''


def test_every_convolution_path_is_checked():
    env = dict(os.environ, NKB_DEBUG_BOUNDS="1")
    r = subprocess.run([sys.executable, "-c", CHILD % ROOT], env=env, capture_output=True,
                       text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "CONV_BOUNDS_OK" in r.stdout, r.stdout[-1500:] + r.stderr[-3000:]
