"""The kernels of small and tall decode projections, the token tiles of the prefill GEMM, and the merge of a step's attention ranges, at the sizes where they change
over: one row, ragged tiles, the first size past one wave, contexts around a range's and a cluster's end."""
from __future__ import annotations

import numpy as np
import pytest

from dooms_b200 import CudaLlamaDecoder, synth
from dooms_b200 import _lib as L
from helpers import launched, rel_l2, write

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHORT_TYPES = [L.F16, L.Q4_0, L.Q5_0, L.Q8_0]
U = 2.0 ** -24


def _matrix(dtype, rows, cols, seed):
    """(block bytes, the values they stand for in f64), both on the GPU."""
    from dooms_b200.quantize import quantize
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = quantize(dtype, torch.randn(rows, cols, device="cuda", generator=gen) * 0.02)
    values = torch.empty(rows, cols, device="cuda")
    L.check(L.lib().dooms_cuda_dequantize(dtype, w.data_ptr(), rows, cols, values.data_ptr(), 0))
    return w, values.double()


def _bound(dtype, values, x):
    """What f32 sums over blocks (f16: over elements, two to four chains a row) and the input's 27 digits below a block's largest allow, row by row."""
    cols = values.shape[1]
    adds = cols / 2 + 32 if dtype == L.F16 else cols / 32 + 32
    largest = x.abs().view(-1, 32).amax(1).repeat_interleave(32).double()
    return adds * U * (values.abs() @ x.abs().double()) + 2 * U * (values.abs() @ largest) + 1e-30


@pytest.mark.parametrize("dtype", SHORT_TYPES)
@pytest.mark.parametrize("rows,cols", [(1, 64), (7, 896), (8, 896), (9, 896), (149, 896), (896, 4864), (1153, 896), (18945, 128), (18977, 896), (28417, 128), (28431, 896), (28417, 4096)])
def test_matvec_of_small_and_tall_matrices(dtype, rows, cols):
    w, values = _matrix(dtype, rows, cols, rows + cols)
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(cols, device="cuda", generator=gen)
    bias = torch.randn(rows, device="cuda", generator=gen)
    y = torch.full((rows,), 0.5, device="cuda")
    names = launched(lambda: L.check(L.lib().dooms_cuda_matvec(dtype, w.data_ptr(), x.data_ptr(), y.data_ptr(), bias.data_ptr(), rows, cols, 2 | 4, 0)))      # y += W x + bias
    # blocks of up to 64 rows, two (f16: three) on each of 148 SMs, 92 KB each at most (64 f16 rows of 896 are more)
    tall = rows > (3 if dtype == L.F16 else 2) * 148 * 64 or (dtype == L.F16 and (rows, cols) == (18977, 896))
    assert not names or ("k_gemv_tall" if tall else "k_gemv_short") in names[0][0]
    ref = values @ x.double()
    err = (y.double() - (ref + bias.double() + 0.5)).abs()
    assert bool((err <= _bound(dtype, values, x) + 4 * U * (ref.abs() + bias.abs().double() + 1)).all())


@pytest.mark.parametrize("rows,cols", [(18977, 896), (28431, 128), (28417, 4096)])
def test_tall_matrix_on_an_input_that_is_already_split(rows, cols):
    w, values = _matrix(L.Q4_0, rows, cols, 41)
    gen = torch.Generator(device="cuda").manual_seed(9)
    x, bias = torch.randn(cols, device="cuda", generator=gen), torch.randn(rows, device="cuda", generator=gen)
    split = torch.empty(L.lib().dooms_cuda_split_input_bytes(cols), dtype=torch.uint8, device="cuda")
    L.check(L.lib().dooms_cuda_split_input(x.data_ptr(), cols, split.data_ptr(), 0))
    y = torch.full((rows,), 0.5, device="cuda")
    names = launched(lambda: L.check(L.lib().dooms_cuda_matvec_split(L.Q4_0, w.data_ptr(), None, split.data_ptr(), y.data_ptr(), bias.data_ptr(), rows, cols, 2 | 4, 0)))
    assert not names or "k_gemv_tall" in names[0][0]
    ref = values @ x.double()
    err = (y.double() - (ref + bias.double() + 0.5)).abs()
    assert bool((err <= _bound(L.Q4_0, values, x) + 4 * U * (ref.abs() + bias.abs().double() + 1)).all())


# (2-norm error against f64 of the f32 dot products on the same matrices and inputs, in the order of _inputs)
F32_DOTS = [(L.Q5_0, 1152, 896, (2.93e-7, 2.98e-7, 2.55e-7, 2.95e-7)), (L.Q8_0, 128, 896, (1.23e-7, 1.18e-7, 1.06e-7, 1.38e-7)),
            (L.Q8_0, 151936, 896, (1.19e-7, 1.16e-7, 1.09e-7, 1.39e-7)), (L.Q6_K, 896, 4864, (2.47e-7, 2.47e-7, 2.85e-7, 2.52e-7))]


def _inputs(cols, seed):
    """What a projection meets: a normalized row; silu(g) * u; elements over orders of magnitude; one in a hundred a thousand times its neighbours."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x, y, z = (torch.randn(cols, device="cuda", generator=gen) for _ in range(3))
    outlier = x.clone()
    outlier[3::97] *= 1000
    return x, torch.nn.functional.silu(2 * x) * y, x * torch.exp(2 * z), outlier


@pytest.mark.parametrize("dtype,rows,cols,f32", F32_DOTS)
def test_the_inputs_digits_cost_no_accuracy(dtype, rows, cols, f32):
    """The input is held in 27 bits below its 32-element block's largest value, its products are exact and a block's sum is rounded once: together no further from f64
    than dot products in f32."""
    w, values = _matrix(dtype, rows, cols, 1)
    worse = [0.0] * 4, [0.0] * 4
    for seed in range(8):
        for i, x in enumerate(_inputs(cols, 100 + seed)):
            y = torch.empty(rows, device="cuda")
            L.check(L.lib().dooms_cuda_matvec(dtype, w.data_ptr(), x.data_ptr(), y.data_ptr(), None, rows, cols, 0, 0))
            ref = values @ x.double()
            worse[0][i] += float(((y.double() - ref) ** 2).sum())
            worse[1][i] += float((ref ** 2).sum())
    errors = [(e / n) ** 0.5 for e, n in zip(*worse)]
    assert all(e <= f for e, f in zip(errors, f32)), errors


@pytest.mark.parametrize("dtype", SHORT_TYPES)
def test_a_bias_that_the_call_before_writes(dtype):
    """y1 = W1 x, then y2 = W2 x2 + y1 on the same stream: the second call may start early, but not read y1 before the first is done. W1 is the larger one, so the
    second is waiting while y1 is being written; in between y1 holds NaN."""
    w1, v1 = _matrix(dtype, 896, 4864, 31)
    w2, v2 = _matrix(dtype, 896, 64, 32)
    gen = torch.Generator(device="cuda").manual_seed(8)
    x1, x2 = torch.randn(4864, device="cuda", generator=gen), torch.randn(64, device="cuda", generator=gen)
    y1, y2 = torch.empty(896, device="cuda"), torch.empty(896, device="cuda")
    ref = v1 @ x1.double() + v2 @ x2.double()
    bound = _bound(dtype, v1, x1) + _bound(dtype, v2, x2) + 4 * U * (v1 @ x1.double()).abs() + 4 * U * ref.abs()
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(300):
        y1.fill_(float("nan"))
        L.check(L.lib().dooms_cuda_matvec(dtype, w1.data_ptr(), x1.data_ptr(), y1.data_ptr(), None, 896, 4864, 0, 0))
        L.check(L.lib().dooms_cuda_matvec(dtype, w2.data_ptr(), x2.data_ptr(), y2.data_ptr(), y1.data_ptr(), 896, 64, 4, 0))
        wrong += (~((y2.double() - ref).abs() <= bound)).sum()
    assert int(wrong) == 0


@pytest.mark.parametrize("dtype", SHORT_TYPES)
@pytest.mark.parametrize("rows,cols", [(1, 64), (32, 896), (4864, 896), (33, 256)])
def test_gate_up_of_small_matrices(dtype, rows, cols):
    wg, vg = _matrix(dtype, rows, cols, 1)
    wu, vu = _matrix(dtype, rows, cols, 2)
    x = torch.randn(cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6)) * 10
    h = torch.empty(rows, device="cuda")
    L.check(L.lib().dooms_cuda_gate_up(dtype, wg.data_ptr(), wu.data_ptr(), x.data_ptr(), h.data_ptr(), rows, cols, 0))
    g, u = vg @ x.double(), vu @ x.double()
    bg, bu = _bound(dtype, vg, x), _bound(dtype, vu, x)
    ref = torch.nn.functional.silu(g) * u
    # silu is 1.1-Lipschitz and at most |g|; exp, divide and the two products round to a few ulp
    assert bool(((h.double() - ref).abs() <= 1.1 * bg * (u.abs() + bu) + g.abs() * bu + 16 * U * ref.abs() + 1e-30).all())


@pytest.mark.parametrize("dtype", SHORT_TYPES + [L.Q4_K, L.Q6_K])
@pytest.mark.parametrize("rows", [64, 18977])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_an_input_that_is_not_finite_is_not_hidden(dtype, rows, bad):
    """One such element: NaN everywhere; an infinity through the kernels of this file as in f32, +-inf by the sign of its weight and NaN where that is zero."""
    cols = 1024 if dtype in (L.Q4_K, L.Q6_K) else 896
    w, values = _matrix(dtype, rows, cols, 3)
    x = torch.randn(cols, device="cuda")
    x[700] = bad
    y = torch.zeros(rows, device="cuda")
    L.check(L.lib().dooms_cuda_matvec(dtype, w.data_ptr(), x.data_ptr(), y.data_ptr(), None, rows, cols, 0, 0))
    assert not bool(torch.isfinite(y).any())
    want = values[:, 700] * bad
    if np.isnan(bad) or dtype in SHORT_TYPES:
        assert bool((torch.isnan(y) == torch.isnan(want)).all())
        assert bool((torch.isnan(want) | (y.double() == want)).all())


@pytest.mark.parametrize("dtype", [L.F16, L.Q4_0, L.Q4_K, L.Q6_K])
@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("tokens,rows,cols", [(1, 128, 256), (63, 130, 512), (65, 896, 1024), (129, 896, 4864), (300, 1152, 768), (513, 300, 512)])
def test_matmul_over_its_token_tiles(dtype, gate, tokens, rows, cols):
    w, values = _matrix(dtype, rows, cols, 11)
    w2, values2 = _matrix(dtype, rows, cols, 12)
    x = torch.randn(tokens, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7)).half()
    y = torch.zeros(tokens, rows, device="cuda")
    L.check(L.lib().dooms_cuda_matmul(dtype, w.data_ptr(), w2.data_ptr() if gate else None, x.data_ptr(), y.data_ptr(), None, tokens, rows, cols, 0, 0))
    L.check(L.lib().dooms_cuda_kernel_status(0, None))
    half = [v.half().double() for v in (values, values2)]      # the tiles hold the weights rounded to f16
    ref = x.double() @ half[0].T
    if gate:
        ref = torch.nn.functional.silu(ref) * (x.double() @ half[1].T)
    # f16 products are exact in f32; the accumulator adds cols / 16 partial sums: 1e-5 covers 4864 of them (measured 6e-6), the gate's product twice that
    assert rel_l2(y.cpu().numpy(), ref.cpu().numpy()) < (2e-5 if gate else 1e-5)


@pytest.mark.parametrize("tokens", [64, 512])
def test_silu_of_a_gate_up_product_is_the_divisions(tokens):
    """One-hot tokens against weights that run through all finite f16 values, and an up matrix of ones: each result is silu of one value. It is
    v / (1 + exp(-v)) in f32 with the division rounded to nearest, but for a last bit here and there; past exp(-v) = 2^126 it may be zero."""
    v = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.float16)
    v = v[torch.isfinite(v)]
    w = v[:v.numel() // 64 * 64].view(-1, 64).cuda().contiguous()
    ones = torch.ones_like(w)
    x = torch.eye(64, dtype=torch.float16, device="cuda").repeat(tokens // 64, 1).contiguous()
    y = torch.empty(tokens, w.shape[0], device="cuda")
    L.check(L.lib().dooms_cuda_matmul(L.F16, w.data_ptr(), ones.data_ptr(), x.data_ptr(), y.data_ptr(), None, tokens, w.shape[0], 64, 0, 0))
    L.check(L.lib().dooms_cuda_kernel_status(0, None))
    got, wf = y.T.reshape(w.shape[0], tokens // 64, 64), w.float()
    want = wf / (1 + torch.exp(-wf))
    small = wf < -87
    for t in range(tokens // 64):
        g = got[:, t]
        assert float((g - want)[small].abs().max()) < 1.1e-36
        ulps = (g.view(torch.int32) - want.view(torch.int32)).abs()[~small]
        assert int(ulps.max()) <= 1 and float((ulps > 0).float().mean()) < 0.01


@pytest.mark.parametrize("position", [62, 126, 254, 510, 1022])
def test_positions_around_a_range_and_a_cluster(tmp_path, position):
    """A step's ranges are 128 keys, the blocks of eight of them merge in shared memory: the logits after one position per call are those of the same tokens in one
    call of a decoder whose prompts stay in f32 (prefill_tile = 1), within the token-by-token bound. A key lost at a range's end moves them by 1e-3 and more."""
    spec = synth.tiny_spec(synth.pure(L.Q8_0), context_length=2048)
    path = write(tmp_path, "ranges", spec, 21)
    ids = [int(t) for t in synth.prompt_tokens(position + 6, spec.n_vocab, 22)]
    dec, f32 = CudaLlamaDecoder.load(path, 1200, 512, prefill_tile=1), CudaLlamaDecoder.load(path, 1200, 512, prefill_tile=1)
    dec.eval_tokens(ids[:position])
    for i, t in enumerate(ids[position:]):
        dec.eval_tokens([t])
        f32.reset()
        f32.eval_tokens(ids[:position + i + 1])
        assert rel_l2(dec.logits(), f32.logits()) < 1e-4, i
