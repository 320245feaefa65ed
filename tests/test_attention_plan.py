"""The plan of the even split over the CTAs, which is host arithmetic: bounds on the contexts of any size."""

from __future__ import annotations

import subprocess
import sys

from conftest import ROOT

PROBE = """
from cross_dsl_kernels_b200 import _native
size = _native.lib().xdk_paged_decode_attention_scratch_bytes
for tokens, q_heads, kv_heads, dim, dtype in ((64, 32, 8, 128, 2), (16, 32, 8, 128, 2), (1, 8, 1, 64, 0), (16384, 65535, 65535, 64, 1)):
    want = size(tokens, q_heads, kv_heads, dim, 2 ** 31, dtype)
    assert want > 0 and want == size(tokens, q_heads, kv_heads, dim, 0, dtype)
    for hint in (2 ** 32, 2 ** 45, 2 ** 53 + 7, 2 ** 60, 2 ** 61, 2 ** 62 - 1, 2 ** 62, 2 ** 63 - 128, 2 ** 63 - 1):
        assert size(tokens, q_heads, kv_heads, dim, hint, dtype) == want, (tokens, kv_heads, hint)
assert size(2 ** 62, 8, 8, 64, 8192, 2) == 0 and size(16, 2 ** 61, 2 ** 61, 64, 8192, 2) == 0
"""


def test_any_bound_on_the_contexts_makes_a_plan():
    """A bound far beyond any cache ("no bound") is one more long context: the same grid, in a process of its own because the
    arithmetic used to wrap to a division by zero."""
    done = subprocess.run([sys.executable, "-c", PROBE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, (done.returncode, done.stderr[-2000:])
