"""Launchers that the C ABI reaches only through a decoder, on their own (tests/kernel_entries.cpp, linked from the library's object files): a product whose reduction
is dealt over several blocks per tile, the norm that adds the shares, and prefill attention over clusters of blocks."""
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


# ---------------------------------------------------------------- on the GPU

@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [L.F16, L.Q4_0, L.Q4_K])
@pytest.mark.parametrize("M,N,K", [(45, 256, 2304), (64, 130, 1024), (129, 300, 4864 // 256 * 256)])
def test_shares_of_a_product_add_up_to_it(entries, dtype, M, N, K):
    """Every count of shares that fits, uneven last ones among them, through the wide producers (q4_0, q4_K: shares of 256 elements) and on f16 rows."""
    from dooms_b200.quantize import quantize
    gen = torch.Generator(device="cuda").manual_seed(M)
    w = quantize(dtype, torch.randn(N, K, device="cuda", generator=gen) * 0.02)
    values = torch.empty(N, K, device="cuda")
    L.check(L.lib().dooms_cuda_dequantize(dtype, w.data_ptr(), N, K, values.data_ptr(), 0))
    rows16 = values.half()
    x = torch.randn(M, K, device="cuda", generator=gen).half()
    ref = x.double() @ rows16.double().T
    # f32 sums over K / 16 MMA steps and the shares
    bound = (K / 16 + 40) * U * (x.double().abs() @ rows16.double().abs().T) + 1e-30
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    for route, units in (("rows16", K // 64), ("gemm", K // 64 if dtype == L.F16 else K // 256)):
        counts = [k for k in range(1, min(units, 32) + 1) if fills(units, k)]
        for k in sorted({1, 2, 3, counts[len(counts) // 2], counts[-2], counts[-1]} & set(counts)):
            shares = torch.full((k, M, N), float("nan"), device="cuda")
            if route == "rows16":
                e = entries.kernel_gemm_rows16(rows16.data_ptr(), x.data_ptr(), shares.data_ptr(), M, N, K, error.data_ptr(), k)
            else:
                e = entries.kernel_gemm(dtype, w.data_ptr(), x.data_ptr(), shares.data_ptr(), M, N, K, error.data_ptr(), None, 0, k)
            assert e == 0, (route, k)
            torch.cuda.synchronize()
            assert int(error) == 0
            assert bool(((shares.double().sum(0) - ref).abs() <= bound).all()), (route, k)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 63, 64, 300])
@pytest.mark.parametrize("E", [64, 896, 1024, 1056, 4096, 5120, 8192, 8224])
@pytest.mark.parametrize("n_shares", [0, 1, 3, 32])
def test_a_norm_adds_the_shares_in_front_of_it(entries, rows, E, n_shares):
    gen = torch.Generator(device="cuda").manual_seed(E)
    x = torch.randn(rows, E, device="cuda", generator=gen)
    gamma = torch.rand(E, device="cuda", generator=gen) + 0.5
    shares = torch.randn(max(1, n_shares), rows, E, device="cuda", generator=gen)
    total = x.double() + shares[:n_shares].double().sum(0)
    size = x.double().abs() + shares[:n_shares].double().abs().sum(0)
    left, out = x.clone(), torch.empty_like(x)
    out16 = torch.empty(rows, E, dtype=torch.float16, device="cuda")
    assert entries.kernel_rms_norm(left.data_ptr(), gamma.data_ptr(), out.data_ptr(), out16.data_ptr(), rows, E, 1e-6, shares.data_ptr(), n_shares) == 0
    torch.cuda.synchronize()
    assert bool(((left.double() - total).abs() <= max(1, n_shares) * U * size).all())
    ref = total / torch.sqrt((total ** 2).mean(1, keepdim=True) + 1e-6) * gamma.double()
    # the sum of squares: E / 1024 + 15 additions in a row; the factor, two products; what the sums of the shares are off
    slack = (E / 1024 + 32) * U * ref.abs() + max(1, n_shares) * U * size * (ref.abs() / total.abs().clamp(min=1e-30))
    assert bool(((out.double() - ref).abs() <= slack).all())
    assert bool(((out16.double() - ref).abs() <= slack + 2.0 ** -11 * ref.abs() + 2.0 ** -25).all())
    # the same sums from the kernel that only adds
    added = x.clone()
    if n_shares:
        assert entries.kernel_add_shares(added.data_ptr(), shares.data_ptr(), n_shares, rows * E) == 0
        torch.cuda.synchronize()
        assert bool(((added.double() - total).abs() <= n_shares * U * size).all())


# position of the first query, queries: one block per query tile; two, four and eight; tiles that end past the chunk; clusters whose last blocks hold no key of the
# first queries
@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim", [(14, 2, 64), (4, 1, 64), (8, 2, 128)])
@pytest.mark.parametrize("pos,M", [(0, 1), (0, 37), (0, 64), (0, 65), (0, 300), (1023, 1), (1024, 130), (2047, 64), (2100, 200), (4095, 33), (5000, 129)])
def test_prefill_attention_over_clusters(entries, heads, kv_heads, dim, pos, M):
    gen = torch.Generator(device="cuda").manual_seed(pos + M)
    keys = pos + M
    qkv = torch.randn(M, (heads + 2 * kv_heads) * dim, device="cuda", generator=gen).half().float()      # (the kernel rounds queries to f16)
    k = torch.randn(keys, kv_heads, dim, device="cuda", generator=gen).half()
    v = torch.randn(keys, kv_heads, dim, device="cuda", generator=gen).half()
    state = torch.zeros(16, dtype=torch.int32, device="cuda")
    state[0] = pos
    out = torch.full((M, heads, dim), float("nan"), device="cuda")
    assert entries.kernel_flash(qkv.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), state.data_ptr(), M, heads, kv_heads, dim, keys) == 0
    torch.cuda.synchronize()
    q = qkv[:, :heads * dim].view(M, heads, dim).double()
    hidden = torch.arange(keys, device="cuda")[None] > pos + torch.arange(M, device="cuda")[:, None]
    for h in range(heads):
        kh, vh = k[:, h // (heads // kv_heads)].double(), v[:, h // (heads // kv_heads)].double()
        p = torch.softmax((q[:, h] @ kh.T / dim ** 0.5).masked_fill(hidden, -float("inf")), 1)
        # probabilities rounded to f16 before the second product (relative 2^-11, or 2^-25 of the largest's share), f32 sums: sum |p| |v| of each
        size = p @ vh.abs()
        bound = 2.0 ** -11 * size + 2.0 ** -25 * p.max(1, keepdim=True).values * vh.abs().sum(0)[None] + 1e-5 * size
        assert bool(((out[:, h].double() - p @ vh).abs() <= bound).all()), h
