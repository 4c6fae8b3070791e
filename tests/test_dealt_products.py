"""Launchers that the C ABI reaches only through a decoder, on their own (tests/kernel_entries.cpp, linked from the library's object files): products whose reduction
is dealt over several blocks per tile."""
from __future__ import annotations

import ctypes as C
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from dooms_b200 import _lib as L
from dooms_b200 import build as B

HERE = Path(__file__).resolve().parent
U = 2.0 ** -24


@pytest.fixture(scope="module")
def entries():
    objects = [B.OBJ / (str(src.relative_to(B.CSRC)).replace("/", "_") + ".o") for src in B.sources() if src.parent.name == "kernels"]
    if not all(o.exists() for o in objects):
        B.build()
    out = HERE / "_build" / "libkernel_entries.so"
    if not out.exists() or out.stat().st_mtime < max(p.stat().st_mtime for p in [HERE / "kernel_entries.cpp", *objects]):
        out.parent.mkdir(exist_ok=True)
        subprocess.run([B.nvcc(), *B.NVCC_FLAGS, "-shared", "-x", "cu", str(HERE / "kernel_entries.cpp"), *[f"-Xlinker={o}" for o in objects], "-o", str(out), "-ldl"],
                       check=True, capture_output=True)
    lib = C.CDLL(str(out))
    P, I, Q = C.c_void_p, C.c_int, C.c_longlong
    lib.kernel_gemm_splits.argtypes = [I, P, I, Q, Q, Q, I]
    lib.kernel_rows16_splits.argtypes = [I, Q, Q, I]
    lib.kernel_gemm.argtypes = [I, P, P, P, I, Q, Q, P, P, Q, I]
    lib.kernel_gemm_rows16.argtypes = [P, P, P, I, Q, Q, P, I]
    lib.kernel_gemm_refuses.argtypes = [I, I, Q, Q, I]
    lib.kernel_rms_norm.argtypes = [P, P, P, P, I, I, C.c_float, P, I]
    lib.kernel_add_shares.argtypes = [P, P, I, Q]
    lib.kernel_flash.argtypes = [P, P, P, P, P, I, I, I, I, I]
    return lib


def fills(units, k):
    per = -(-units // k)
    return -(-units // per) == k


def test_a_count_of_shares_that_the_reduction_does_not_divide_into_is_refused(entries):
    """A share that no block writes would be added by the norm all the same."""
    if torch.cuda.is_available():
        pytest.skip("the refusal comes before any use of the device; where there is one, nothing is tried that might be launched")
    for units in (9, 36, 76, 224):
        for k in range(2, 41):
            if k > 32 or not fills(units, k):
                assert entries.kernel_gemm_refuses(L.F16, 1, 256, units * 64, k), (units, k)
                assert entries.kernel_gemm_refuses(L.F16, 0, 256, units * 64, k), (units, k)
                assert entries.kernel_gemm_refuses(L.Q4_0, 0, 256, units * 256, k), (units, k)
                assert entries.kernel_gemm_refuses(L.Q4_K, 0, 256, units * 256, k), (units, k)
    assert entries.kernel_gemm_refuses(L.Q5_0, 0, 256, 2048, 2)      # no scratch for its rows: that route deals nothing


def test_planned_counts_of_shares_divide_the_reduction(entries):
    for M in (1, 2, 16, 64, 65, 128, 300, 512, 2048):
        for N, K in ((896, 896), (896, 4864), (256, 2304), (4096, 4096), (4096, 14336), (5120, 27648), (64, 64), (130, 320)):
            for most in (1, 2, 3, 7, 32, 100):
                k = entries.kernel_rows16_splits(M, N, K, most)
                assert 1 <= k <= min(most, 32) and fills(K // 64, k)
                if K % 256 == 0:
                    k = entries.kernel_gemm_splits(L.Q4_0, None, M, N, K, 0, most)
                    assert 1 <= k <= min(most, 32) and fills(K // 256, k)


def planned(env):
    """gemm_tc_k_splits in a process with these switches: (dtype, tokens, bytes of scratch) -> shares of a 256 x 2304 product."""
    cases = [(L.Q4_0, 45, 0), (L.Q4_K, 100, 0), (L.Q4_0, 300, 1 << 30), (L.Q8_0, 45, 1 << 30), (L.Q5_0, 300, 1 << 30), (L.F16, 45, 0)]
    code = ("import ctypes as C, sys; lib = C.CDLL(sys.argv[1]); lib.kernel_gemm_splits.argtypes = [C.c_int, C.c_void_p, C.c_int, C.c_longlong, C.c_longlong, C.c_longlong, C.c_int]; "
            f"print([lib.kernel_gemm_splits(dt, None, m, 256, 2304, b, 32) for dt, m, b in {cases}])")
    r = subprocess.run([sys.executable, "-c", code, str(HERE / "_build" / "libkernel_entries.so")], env={**os.environ, **env}, capture_output=True, text=True, check=True)
    return dict(zip([(dt, m) for dt, m, _ in cases], json.loads(r.stdout)))


def test_the_switches_of_dealt_products(entries):
    plain = planned({})
    assert all(k > 1 for k in plain.values()), plain
    off = planned({"DOOMS_GEMM_SPLIT_K": "0"})
    assert set(off.values()) == {1}, off
    never = planned({"DOOMS_GEMM_PRE_FROM": "100000"})      # no quantized product on f16 rows: q5_0 and q8_0 have no other route that deals one
    assert never[L.Q8_0, 45] == never[L.Q5_0, 300] == 1 and never[L.Q4_0, 45] == plain[L.Q4_0, 45] and never[L.F16, 45] == plain[L.F16, 45], never
