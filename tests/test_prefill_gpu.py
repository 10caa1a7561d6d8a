"""The tcgen05 prefill matmul on a B200: weights rounded once to bf16, one fp32 chain over K; rows do not depend on how
the prompt is chunked.  Mirrors the reference's contract for ``prefill_matmul`` (cuda/kernels/qmm.py:160-171)."""

import numpy as np
import pytest
import torch

from oracle import affine as oaff
from tensorfold_b200 import _lib, synthetic
from tensorfold_b200.cuda.kernels import qmm

from gpu_util import DEV, to_dev

pytestmark = pytest.mark.gpu


def reference(x, words, scales, biases, gs):
    """float64 x @ bf16(q * s + b).T: the weight is rounded once to bf16 (q * s + b is exact in float64)."""

    w = oaff.dequantize(words.numpy(), scales.float().numpy(), biases.float().numpy(), 4, gs)
    w = oaff.bf16_round(w.astype(np.float32)).astype(np.float64)
    return x.float().numpy().astype(np.float64) @ w.T


@pytest.mark.parametrize("n,k,gs,m", [(128, 64, 64, 8), (128, 256, 64, 256), (1024, 5120, 64, 300), (384, 2048, 32, 70),
                                      (200, 1024, 32, 1), (5120, 6144, 64, 512)])
def test_matches_the_oracle(n, k, gs, m):
    w = synthetic.affine_weight(n, k, 4, gs, seed=n + k + m)
    q = qmm.pack(*to_dev(*w), gs)
    x = synthetic.activations(m, k, 1)
    y = qmm.prefill_matmul(x.to(DEV), q)
    assert y.shape == (m, n) and y.dtype == torch.bfloat16
    ref = reference(x, *w, gs)
    err = np.abs(y.float().cpu().numpy() - ref).max()
    assert err <= np.abs(ref).max() * 2 ** -7, f"max abs error {err} vs {np.abs(ref).max()}"
    f32 = qmm.prefill_matmul(x.to(DEV), q, f32=True)
    assert torch.equal(f32.to(torch.bfloat16), y)
    assert np.abs(f32.cpu().numpy() - ref).max() <= np.abs(ref).max() * 2 ** -12
    assert _lib.device_error(y) == 0


@pytest.mark.parametrize("n,k,gs,m", [(1, 64, 64, 17), (136, 192, 64, 193), (257, 128, 64, 385), (392, 320, 32, 16), (1160, 704, 64, 130)])
def test_edges_of_the_paired_tiles(n, k, gs, m):
    """Columns past one block of a pair and past 8, an odd number of 128-column blocks, rows one past a tile of 16, 128 or
    192, and K that ends with half of a 128-input stage; the oracle and the tolerance of the test above."""

    w = synthetic.affine_weight(n, k, 4, gs, seed=n + m)
    q = qmm.pack(*to_dev(*w), gs)
    x = synthetic.activations(m, k, 4)
    ref = reference(x, *w, gs)
    f32 = qmm.prefill_matmul(x.to(DEV), q, f32=True)
    assert np.abs(f32.cpu().numpy() - ref).max() <= np.abs(ref).max() * 2 ** -12
    wide = torch.full((m, n + 8), 7.0, dtype=torch.bfloat16, device=DEV)                  # a slice of wider rows as output
    y = qmm.prefill_matmul(x.to(DEV), q, out=wide[:, :n])
    assert torch.equal(y, f32.to(torch.bfloat16)) and bool((wide[:, n:] == 7.0).all())
    assert _lib.device_error(y) == 0


@pytest.mark.parametrize("act", ["swiglu", "relu2"])
@pytest.mark.parametrize("k,m", [(96, 33), (160, 200)])
def test_epilogues_at_the_edges(act, k, m):
    """K ends inside a half stage (groups of 32); the epilogue works on the bf16 of the plain product's sums."""

    gs, half = 32, 144
    a, b = (synthetic.affine_weight(half, k, 4, gs, seed=s) for s in (5, 6))
    q = qmm.pack_pair(to_dev(*a), to_dev(*b), gs)
    x = synthetic.activations(m, k, 8).to(DEV)
    got = qmm.matmul_act(x, q, act=act, prefill=True).float()
    v = torch.from_numpy(np.concatenate([reference(x.cpu(), *w, gs) for w in (a, b)], 1)).to(torch.bfloat16).double()
    gate, up = v[:, :half], v[:, half:]
    if act == "swiglu":
        want = (gate / (1 + torch.exp(-gate))).to(torch.bfloat16).double() * up
    else:
        want = torch.stack([gate.view(m, 9, 16), up.view(m, 9, 16)], 2).view(m, 2 * half).clamp(min=0) ** 2
    # a factor may round to the neighbouring bf16 value (2^-8 relative each), the product rounds once more
    assert (got.cpu().double() - want).abs().max() <= want.abs().max() * 3 * 2 ** -8
    assert _lib.device_error(x) == 0


@pytest.mark.parametrize("act", [None, "relu2"])
def test_weights_the_previous_kernel_wrote(act):
    """A prompt matmul writes the packed units (as bf16 rows) that the next one multiplies with, and nothing waits in
    between: its blocks run on few SMs for long, and signal their dependents at once."""

    n, kg, gs = 2048, 8, 64
    q1 = qmm.pack(*to_dev(*synthetic.raw_weight(2304, 16384, 4, 64, 1)), 64)
    x1 = synthetic.activations(n // 128 * kg, 16384, 2).to(DEV)
    x2 = synthetic.activations(48, kg * gs, 3).to(DEV)
    units = torch.zeros((n // 128, kg, 1152), dtype=torch.int32, device=DEV)
    q2 = qmm.Q4(units, None, None, n, kg * gs, gs)
    run = lambda: qmm.prefill_matmul(x2, q2, f32=True) if act is None else qmm.matmul_act(x2, q2, act=act, prefill=True)
    for _ in range(3):
        units.zero_()
        torch.cuda.synchronize()
        qmm.prefill_matmul(x1, q1, out=units.view(torch.bfloat16).view(-1, 2304))
        got = run()
        torch.cuda.synchronize()
        want = run()
        assert torch.isfinite(want).all() and want.any()
        assert torch.equal(got, want)


def test_exact_integer_case_is_bit_exact():
    rng = np.random.default_rng(7)
    n, k, gs, m = 140, 128, 64, 19
    values = rng.integers(0, 16, size=(n, k), dtype=np.uint32)
    words = torch.from_numpy(oaff.pack_codes(values, 4).view(np.int32))
    scales, biases = torch.full((n, 2), 0.25).bfloat16(), torch.full((n, 2), -0.5).bfloat16()
    xf = rng.integers(-2, 3, size=(m, k)).astype(np.float32) * 0.5
    want = np.sum(xf[:, None, :] * (values.astype(np.float32) * 0.25 - 0.5)[None, :, :], axis=2)
    q = qmm.pack(*to_dev(words, scales, biases), gs)
    got = qmm.prefill_matmul(torch.from_numpy(xf).bfloat16().to(DEV), q, f32=True)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("n,k,gs", [(1024, 5120, 64), (512, 2048, 32)])
def test_rows_do_not_depend_on_the_chunk(n, k, gs):
    q = qmm.pack(*to_dev(*synthetic.raw_weight(n, k, 4, gs, 3 * n + k)), gs)
    x = synthetic.activations(700, k, 5).to(DEV)
    whole = qmm.prefill_matmul(x, q)
    for a, b in ((0, 1), (255, 257), (699, 700), (0, 256), (100, 612), (3, 4)):
        assert torch.equal(qmm.prefill_matmul(x[a:b], q), whole[a:b]), (a, b)
    perm = torch.randperm(700, generator=torch.Generator().manual_seed(3)).to(DEV)
    assert torch.equal(qmm.prefill_matmul(x[perm], q), whole[perm])
    wide = torch.zeros((700, k + 64), dtype=torch.bfloat16, device=DEV)
    wide[:, :k] = x
    assert torch.equal(qmm.prefill_matmul(wide[:, :k], q), whole)             # strided rows


def test_blocks_that_run_several_tiles_keep_the_bits():
    """360 tiles on at most 148 persistent blocks: a block runs two or three tiles back to back on alternating
    accumulators.  Every 256-row chunk run on its own (40 tiles: one per block) must give the same bits, and the whole
    must match the oracle."""

    n, k, gs, m = 5120, 256, 64, 2304
    w = synthetic.affine_weight(n, k, 4, gs, seed=77)
    q = qmm.pack(*to_dev(*w), gs)
    x = synthetic.activations(m, k, 9)
    whole = qmm.prefill_matmul(x.to(DEV), q)
    for a in range(0, m, 256):
        assert torch.equal(qmm.prefill_matmul(x[a:a + 256].to(DEV), q), whole[a:a + 256]), a
    ref = reference(x, *w, gs)
    assert np.abs(whole.float().cpu().numpy() - ref).max() <= np.abs(ref).max() * 2 ** -7
    pair = qmm.pack_pair(to_dev(*w), to_dev(*synthetic.affine_weight(n, k, 4, gs, seed=78)), gs)
    act = qmm.matmul_act(x.to(DEV), pair, act="swiglu", prefill=True)       # 80 x 9 tiles through the SwiGLU drain
    for a in (0, 1024, 2048):
        assert torch.equal(qmm.matmul_act(x[a:a + 256].to(DEV), pair, act="swiglu", prefill=True), act[a:a + 256]), a
    assert _lib.device_error(whole) == 0


def test_other_formats_fall_back_to_the_exact_matmul():
    w = synthetic.affine_weight(256, 1024, 3, 128, seed=4)
    q = qmm.pack(*to_dev(*w), 128, bits=3)
    x = synthetic.activations(40, 1024, 2).to(DEV)
    assert torch.equal(qmm.prefill_matmul(x, q), qmm.matmul(x, q))
