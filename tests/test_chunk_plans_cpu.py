"""The chunk rule on the host: its plans' invariants (tests/even_chunk_props.cpp),
and the float32 phase of a mixed solve, which brings its own workspace, in the
rule's chunks at every size."""

import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parallel-in-time-ode-filters_gb300", "csrc")


def test_even_chunks_hold_their_invariants(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "even_chunk_props")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(ROOT, "tests", "even_chunk_props.cpp"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr


@pytest.mark.parametrize("n,D,d", [(131500, 3, 1), (18200, 6, 2), (8700, 9, 3), (5000, 8, 2)])
def test_mixed_solve_takes_the_rule_for_both_phases(n, D, d, monkeypatch):
    """With either chunk length the float32 pass of these sizes lies on both
    sides of 16 MiB, a limit that only the allocation-free pass has."""
    from pof import _lib

    lib = _lib.lib()
    lanes = 1 if D < 6 else (8 if D <= 8 else 16)
    target = 19456 if lanes == 1 else 48640 // lanes
    c = max(-(-n // target), 4 if lanes == 1 else 2)
    dflt = lib.pof_ieks_mixed_workspace_bytes(ctypes.c_int64(n), D, d)
    monkeypatch.setenv("POF_C0", str(c))
    assert lib.pof_ieks_mixed_workspace_bytes(ctypes.c_int64(n), D, d) == dflt > 0
