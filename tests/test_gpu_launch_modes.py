"""Q27_PDL is read once in a process: unset, the kernels of a decode step start while their predecessor drains; 1, every
kernel may; 0, none does. The suite runs with it unset; here the tests that depend on the order of wait and trigger run with
the other two values, in a process of their own (all split-K kernels, chunks that are left unwritten, capture behind copies
and joins, two streams, the paged batch, the prologue and a prefill behind it)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SUBSET = ["tests/test_gpu_decode.py::" + t for t in (
    "test_config1_cpu_checkable", "test_decode_head_counts", "test_q8_1_epilogue", "test_empty_chunks_leave_no_trace",
    "test_partial_of_a_short_slice_has_no_trace", "test_step_captured_behind_a_copy_and_another_stream",
    "test_steps_on_two_streams_of_the_caller", "test_kv_length_partials_merge")] + [
    "tests/test_gpu_paged.py::test_paged_batched_decode", "tests/test_gpu_paged.py::test_prep_paged_equals_prep_per_sequence",
    "tests/test_gpu_kv_append.py::test_attn_prep", "tests/test_gpu_prefill.py::test_prefill_split_kv",
    "tests/test_gpu_prefill.py::test_prefill_q8_1_epilogue"]


@pytest.mark.parametrize("mode", ["0", "1"])
def test_other_launch_modes(q27, mode):
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider"] + SUBSET, cwd=ROOT,
                       env=dict(os.environ, Q27_PDL=mode), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
    assert " passed" in r.stdout
