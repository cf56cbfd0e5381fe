"""The planners' measurement hooks, which only a tuning build exports."""
import ctypes
import os
import subprocess

import pytest

from kungfu_b200.csrc import build


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    try:
        nvcc = build.find_nvcc()
    except build.BuildError as e:
        pytest.skip(str(e))
    out = str(tmp_path_factory.mktemp("tuning") / "planner.so")
    files = [os.path.join(build.HERE, f) for f in ("attention_prefill_tc.cu", "runtime.cu")]
    subprocess.run([nvcc, *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-DKF_TUNING", "-shared", "-o", out, *files], check=True, capture_output=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("parts,run_tiles,planned", [(3, 0, -2), (1, 0, -2), (2, 16, 16)])
def test_a_fixed_plan_of_prompt_attention(lib, parts, run_tiles, planned):
    """Run tiles 0 cuts every tile, which the caller must be able to tell from a planner's 0 (short tiles may stay whole)."""
    got = ctypes.c_int(0)
    lib.kf_set_attention_prefill_plan(parts, run_tiles)
    try:
        assert lib.kf_attention_prefill_tc_plan(4, 8, 8192, ctypes.byref(got)) == parts
        assert got.value == planned
    finally:
        lib.kf_set_attention_prefill_plan(0, 0)
