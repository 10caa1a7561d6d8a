"""The tensor-memory kernel for more than 16 rows (tf_qmm_window) on a B200: every row must carry the bits the tiled kernel
gives, at the edges of its row tiles (16, 32, 48, 64, 256), with one and several K slices, odd column counts, and all formats."""

import pytest
import torch

from tensorfold_b200 import _lib, synthetic
from tensorfold_b200.cuda.kernels import qmm

from gpu_util import DEV, to_dev

pytestmark = pytest.mark.gpu


def packed(n, k, gs, bits=4):
    return qmm.pack(*to_dev(*synthetic.raw_weight(n, k, bits, gs, n + 3 * k)), gs, bits=bits)


def tiled(monkeypatch, x, q, xs=None, **kw):
    with monkeypatch.context() as m:
        m.setattr(qmm, "STREAM", False)
        return qmm.matmul(x, q, xs, **kw)


def window(x, q, xs=None, *, sk, f32=False, out=None):
    """The call through tf_qmm_window, whatever kernel matmul would pick for its size."""

    lib, m = _lib.lib(), x.shape[0]
    if out is None:
        out = torch.empty((m, q.n), dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
    need = lib.tf_qmm_window_part_bytes(m, q.n, q.bits, sk)
    assert need >= 0
    part, count = torch.empty((max(need, 16),), dtype=torch.uint8, device=DEV), torch.zeros((65536,), dtype=torch.uint8, device=DEV)
    rc = lib.tf_qmm_window(x.data_ptr(), x.stride(0), m, None if xs is None else xs.data_ptr(), q.weight.data_ptr(),
                           q.weight.stride(0), q.n, q.k, q.bits, q.gs, sk, out.data_ptr(), out.stride(0), int(f32),
                           count.data_ptr(), count.numel(), part.data_ptr(), need, 0, _lib.stream_of(x))
    _lib.check(rc, "window")
    assert not count.any(), "counters are left at zero"
    return out


@pytest.mark.parametrize("n,k,gs,sk", [(128, 64, 64, 1), (328, 64 * 21, 64, 1), (1000, 64 * 13, 64, 5), (1, 512, 128, 2),
                                       (5120, 6144, 64, 14), (300, 32 * 21, 32, 3), (640, 32 * 7, 32, 1)])
def test_rows_carry_the_tiled_kernels_bits(monkeypatch, n, k, gs, sk):
    q, x = packed(n, k, gs), synthetic.activations(600, k, 4).to(DEV)
    want = tiled(monkeypatch, x, q, sk=sk, f32=True)
    for m in (1, 17, 31, 33, 48, 49, 64, 65, 97, 255, 256, 257, 600):
        assert torch.equal(window(x[:m], q, sk=sk, f32=True), want[:m]), f"rows differ at M={m}"
    xs = qmm.group_sums(x[:70], gs)
    assert torch.equal(window(x[:70], q, xs, sk=sk), tiled(monkeypatch, x[:70], q, xs, sk=sk))
    wide = torch.zeros((40, n + 24), dtype=torch.bfloat16, device=DEV)
    window(x[:40], q, sk=sk, out=wide[:, 8:n + 8])
    assert torch.equal(wide[:, 8:n + 8], want[:40].to(torch.bfloat16)) and not wide[:, :8].any() and not wide[:, n + 8:].any()
    assert _lib.device_error(x) == 0


@pytest.mark.parametrize("bits", [b for b in qmm.BITS if b != 8])
@pytest.mark.parametrize("gs", qmm.GROUPS)
def test_every_format(monkeypatch, bits, gs):
    q, x = packed(328, gs * 13, gs, bits), synthetic.activations(64, gs * 13, 5).to(DEV)
    for m, sk in ((17, 1), (40, 3), (64, 2)):
        assert torch.equal(window(x[:m], q, sk=sk, f32=True), tiled(monkeypatch, x[:m], q, sk=sk, f32=True))


def hard(kind, m, k):
    """Rows whose 16-input steps a differently aligned or truncating adder would round to other bits."""

    g = torch.Generator().manual_seed(len(kind) * 1000 + k)
    x = torch.randn((m, k), generator=g)
    powers = lambda lo, hi: torch.exp2(torch.randint(lo, hi, (m, k), generator=g).float())
    if kind == "spread":                                     # exponents over 60 and over 200 binades
        x[: m // 2] *= powers(-30, 31)[: m // 2]
        x[m // 2:] *= powers(-100, 101)[m // 2:]
    elif kind == "cancelling":                               # v, -v beside much smaller terms, next to each other and apart
        x = (x * powers(-8, 9)).bfloat16().float()
        big = (torch.randn((m, k // 2), generator=g) * 2 ** 20).bfloat16().float() * (torch.rand((m, k // 2), generator=g) < 0.3)
        x[:, 0::2] = torch.where(big != 0, big, x[:, 0::2])
        x[:, 1::2] = torch.where(big != 0, -big, x[:, 1::2])
        x[1::2] = x[1::2, torch.randperm(k, generator=g)]
    elif kind == "subnormal":
        x[: m // 2] *= 2.0 ** -128
        x[m // 2:] *= powers(-133, -100)[m // 2:]
    elif kind == "large":                                    # sums past the largest finite value
        x *= 2.0 ** 118
    elif kind == "zeros":
        x = torch.where(torch.rand((m, k), generator=g) < 0.5, -0.0, 0.0)
        x[: m // 2] = -0.0
    else:                                                    # infinities and NaN here and there
        r = torch.rand((m, k), generator=g)
        x[r < 0.0005], x[(r > 0.0005) & (r < 0.001)], x[r > 0.9997] = float("inf"), -float("inf"), float("nan")
    return x.to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("kind", ["spread", "cancelling", "subnormal", "large", "zeros", "infinite"])
@pytest.mark.parametrize("bits,gs", [(2, 128), (3, 32), (4, 32), (4, 64), (4, 128), (5, 64), (6, 128)])
def test_sums_that_are_hard_to_round_carry_the_same_bits(monkeypatch, kind, bits, gs):
    """Rows keep their bits between up to 16 (persistent kernel), 32 and more rows, which run on mma.sync and on tcgen05.mma:
    their accumulation steps must round alike for every input.  A NaN is a NaN, whatever its bits."""

    q, x = packed(328, gs * 13, gs, bits), hard(kind, 64, gs * 13)
    bits_of = lambda t: t.masked_fill(t.isnan(), 0).view(torch.int32)
    same = lambda a, b: torch.equal(a.isnan(), b.isnan()) and torch.equal(bits_of(a), bits_of(b))
    for m, sk in ((40, 1), (64, 3)):
        want = tiled(monkeypatch, x[:m], q, sk=sk, f32=True)
        assert same(window(x[:m], q, sk=sk, f32=True), want)
        assert same(qmm.matmul(x[:16], q, sk=sk, f32=True), want[:16])


@pytest.mark.parametrize("captured", [False, True])
def test_a_chain_of_calls_with_pdl(monkeypatch, captured):
    """Each call reads the rows the one before it writes, starts before that one has ended, and shares its counters."""

    n = 4096
    qs, x = [packed(n, n, 64), packed(n, n, 64, 3)], synthetic.activations(48, n, 6, std=2 ** -10).to(DEV)
    outs = [torch.zeros((48, n), dtype=torch.bfloat16, device=DEV) for _ in range(6)]

    def chain(matmul, outs, **kw):
        for i, out in enumerate(outs):
            matmul(outs[i - 1] if i else x, qs[i % 2], sk=4, out=out, **kw)

    want = [torch.zeros_like(out) for out in outs]
    chain(lambda *a, **kw: tiled(monkeypatch, *a, **kw), want)
    chain(qmm.matmul, outs, pdl=True)
    if captured:
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain(qmm.matmul, outs, pdl=True)
        for _ in range(3):
            for out in outs:
                out.zero_()
            graph.replay()
    assert all(out.isfinite().all() and torch.equal(out, ref) for out, ref in zip(outs, want)) and outs[-1].any()
    assert _lib.device_error(x) == 0


@pytest.mark.parametrize("n,k,m", [(4096, 4096, 32), (4096, 4096, 33), (4095, 4096, 64), (1024, 5120, 192), (1024, 5120, 256)])
def test_matmul_gives_the_same_bits_on_both_sides_of_its_rule(monkeypatch, n, k, m):
    q, x = packed(n, k, 64), synthetic.activations(m, k + 8, 7).to(DEV)[:, :k]
    assert torch.equal(qmm.matmul(x, q), tiled(monkeypatch, x, q))


@pytest.mark.parametrize("n,k,gs,sk", [(1536, 4096, 64, 10), (1536, 4096, 64, 11), (3072, 5120, 32, 16), (3072, 5120, 32, 17),
                                       (2048, 8192, 64, 22), (2048, 8192, 64, 23), (4096, 8192, 64, 33)])
@pytest.mark.parametrize("m", [192, 257])
def test_matmul_gives_the_same_bits_on_both_sides_of_the_lines_for_slices(monkeypatch, n, k, gs, sk, m):
    q, x = packed(n, k, gs), synthetic.activations(m, k, 7).to(DEV)
    want = tiled(monkeypatch, x, q, sk=sk)
    assert torch.equal(qmm.matmul(x, q, sk=sk), want)
    assert torch.equal(qmm.matmul(x, q, qmm.group_sums(x, gs), sk=sk), want)


def test_graphs_own_their_counters_and_take_no_scratch_area():
    """Graphs captured on one fresh stream replay side by side, and leave the sets' scratch areas to the sets."""

    q, x = packed(4096, 4096, 64), synthetic.activations(48, 4096, 6).to(DEV)
    want, areas = qmm.matmul(x, q, sk=4), len(qmm._set_scratch)
    torch.cuda.synchronize()
    stream, graphs, outs = torch.cuda.Stream(), [torch.cuda.CUDAGraph() for _ in range(2)], [torch.zeros_like(want) for _ in range(2)]
    for graph, out in zip(graphs, outs):
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(4):
                qmm.matmul(x, q, sk=4, out=out)
    assert len(qmm._set_scratch) == areas
    sides = [torch.cuda.Stream() for _ in graphs]
    for _ in range(3):
        for graph, side in zip(graphs, sides):
            with torch.cuda.stream(side):
                graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(out, want) for out in outs) and _lib.device_error(x) == 0


def test_a_capture_zeroes_its_counters_once():
    """Each further call of a capture is one node, its kernel."""

    from cuda.bindings import runtime

    q, x = packed(4096, 4096, 64), synthetic.activations(48, 4096, 6).to(DEV)
    out = qmm.matmul(x, q, sk=4)

    def nodes(calls):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            for _ in range(calls):
                qmm.matmul(x, q, sk=4, out=out)
        return runtime.cudaGraphGetNodes(graph.raw_cuda_graph(), 0)[-1]

    assert nodes(4) - nodes(1) == 3
