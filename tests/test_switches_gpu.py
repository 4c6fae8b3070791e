"""The environment switches of the prefill GEMM's cut, of prefill attention's clusters and of the decode attention's: each leaves the answer where it was and does
what its name says. A switch is read once per process, so every setting runs this file in a process of its own, on one small one-layer model (with one
layer, a sum in another order moves the logits by the f16 roundings it flips and no more)."""
from __future__ import annotations

import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

if __name__ == "__main__":
    sys.path[:0] = [str(Path(__file__).resolve().parent.parent), str(Path(__file__).resolve().parent)]
from dooms_b200 import CudaLlamaDecoder, synth
from dooms_b200 import _lib as L
from helpers import launched, rel_l2, write

pytestmark = pytest.mark.gpu

N_CTX, N_BATCH = 4416, 512      # (69 key tiles: the decode attention's grid is a multiple of eight ranges only when it runs in clusters)
STOPS = [45, 345, 1200, 2300, 4300]      # prompt ends: one wide-producer tile; f16 rows; 10, 18 and 34 key tiles: clusters of 2, 4 and 8
STEPS = {345, 4300}                      # three positions of one call each after these: a handful of ranges, all of them
# A flipped rounding moves an operand by 2^-11 of itself; sums in another order (1e-6 of themselves) flip about one in five hundred of each product's operands:
# 5e-4 * sqrt(1 / 500) = 2e-5 a product, four of them in a row in front of the logits.
FLIPS = 1e-4
# Prefill attention rounds probabilities to f16 relative to the largest score so far, which depends on the cut: 2e-4 of its output on either side (one key lost of
# 4300 moves that by 1 / sqrt(4300) = 1.5e-2).
CUTS = 1e-3


def answers(path: str, **kw):
    """{name: logits} of the prompts and steps, and the kernels they launched."""
    dec = CudaLlamaDecoder.load(path, N_CTX, N_BATCH, **kw)
    ids = [int(t) for t in synth.prompt_tokens(N_CTX, 50, 77)]
    out = {}

    def run():
        at = 0
        for stop in STOPS:
            dec.eval_tokens(ids[at:stop])
            at = stop
            out[f"prompt_{stop}"] = np.asarray(dec.logits())
            for t in range(3 if stop in STEPS else 0):
                dec.eval_tokens([ids[at]])
                at += 1
                out[f"step_{at}"] = np.asarray(dec.logits())
    kernels = launched(run)
    dec.close()
    return out, kernels


@pytest.fixture(scope="module")
def model(model_dir):
    return write(model_dir, "switches", synth.tiny_spec(synth.pure(L.Q4_0), n_layer=1, context_length=N_CTX), 51)


def with_switches(model, tmp_path, **env):
    out = tmp_path / "answers.npz"
    r = subprocess.run([sys.executable, __file__, model, str(out)], env={**os.environ, **env}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = dict(np.load(out))
    return got, json.loads(str(got.pop("kernels")))


@pytest.fixture(scope="module")
def plain(model, tmp_path_factory):
    return with_switches(model, tmp_path_factory.mktemp("plain"))


def grids(kernels, name):
    return [grid for n, grid in kernels if name in n]


def test_the_plain_answers_are_those_of_f32_projections(model, plain):
    """prefill_tile = 1 takes none of these kernels. 1e-2: the bound of weights that are not exact in f16 through the tensor-core tiles."""
    want, _ = answers(model, prefill_tile=1)
    for name, logits in plain[0].items():
        assert rel_l2(logits, want[name]) < 1e-2, name


def test_the_plain_run_reaches_what_the_switches_turn_off(plain):
    kernels = plain[1]
    if not kernels:
        pytest.skip("the profiler lists no kernels here")
    gemm = grids(kernels, "k_gemm_tc")
    assert any(g[2] > 1 for g in gemm[:4]) and any(g[2] > 1 for g in gemm[4:])      # reductions dealt by the wide producers (45 tokens) and on f16 rows (300)
    assert {g[2] for g in grids(kernels, "k_attention_flash")} == {1, 2, 4, 8}
    assert {g[1] % 8 for g in grids(kernels, "k_attention_decode")} == {0}


SWITCHES = [{"DOOMS_GEMM_SPLIT_K": "0"}, {"DOOMS_FLASH_PARTS": "1"}, {"DOOMS_FLASH_PARTS": "2"}, {"DOOMS_ATTN_CLUSTER": "0"}, {"DOOMS_GEMM_TOKENS": "64"},
            {"DOOMS_GEMM_TOKENS": "128"}, {"DOOMS_GEMM_TOKENS": "256"}, {"DOOMS_GEMM_PAIR": "1", "DOOMS_GEMM_TOKENS": "256"}, {"DOOMS_GEMM_PRE_FROM": "16"}]


@pytest.mark.parametrize("env", SWITCHES, ids=lambda e: " ".join(f"{k[6:]}={v}" for k, v in e.items()))
def test_a_switch_leaves_the_answer(model, plain, tmp_path, env):
    got, kernels = with_switches(model, tmp_path, **env)
    for name, want in plain[0].items():
        assert rel_l2(got[name], want) < (CUTS if "DOOMS_FLASH_PARTS" in env else FLIPS), name
    if not kernels:
        return
    if "DOOMS_GEMM_SPLIT_K" in env:
        assert {g[2] for g in grids(kernels, "k_gemm_tc")} == {1}
    if "DOOMS_FLASH_PARTS" in env:
        assert max(g[2] for g in grids(kernels, "k_attention_flash")) == int(env["DOOMS_FLASH_PARTS"])
    if "DOOMS_ATTN_CLUSTER" in env:
        assert all(g[1] % 8 for g in grids(kernels, "k_attention_decode"))


if __name__ == "__main__":
    result, listed = answers(sys.argv[1])
    np.savez(sys.argv[2], kernels=json.dumps(listed), **result)
