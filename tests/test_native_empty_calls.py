"""C entry points with nothing to do: rows but no columns, tokens but no heads.  They return without
a launch, so no GPU is needed; a division by the number of column tiles would end the process, so
each call is made by a child."""

import os
import subprocess
import sys

import pytest

from bitscom_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALLS = {
    "colsum_strips": ("lib.bcom_colsum_strips(ll(5), 0)", 1),
    "colsum": ("lib.bcom_colsum_bf16(z, z, z, ll(5), 0, z)", 0),
    "bias_gelu_fwd": ("lib.bcom_bias_gelu_fwd(z, z, z, ll(5), 0, z)", 0),
    "bias_gelu_bwd": ("lib.bcom_bias_gelu_bwd(z, z, z, z, z, ll(5), 0, z)", 0),
    "rope": ("lib.bcom_rope(z, z, z, ll(5), 0, 64, ll(64), 128, 0, z)", 0),
    "rope_head_dim": ("lib.bcom_rope(z, z, z, ll(5), 4, 0, ll(64), 128, 0, z)", 0),
    "rope_no_positions": ("lib.bcom_rope(z, z, z, ll(5), 4, 64, ll(256), 0, 0, z)", 1),
    "rope_copy": ("lib.bcom_rope_copy(z, z, z, z, ll(5), 0, 64, ll(64), 0, 128, 1, z)", 0),
}


@pytest.mark.skipif(_build.nvcc_path() is None and not os.path.exists(
    _build.lib_path("bcom_llama")), reason="needs the built library")
@pytest.mark.parametrize("name", sorted(CALLS))
def test_empty_call_returns(name):
    call, want = CALLS[name]
    code = ("import ctypes\n"
            "from bitscom_b200 import _build\n"
            "lib = _build.load_library('bcom_llama')\n"
            "z, ll = ctypes.c_void_p(0), ctypes.c_longlong\n"
            f"print('rc', {call})\n")
    run = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         timeout=600)
    assert run.returncode == 0, (run.returncode, run.stderr[-500:])
    assert run.stdout.split()[-2:] == ["rc", str(want)]
