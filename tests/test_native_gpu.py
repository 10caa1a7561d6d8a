"""The host path (``csrc/native.cpp``) on a B200: who owns the memory a launch was given."""

import ctypes
import subprocess

import pytest
import torch

from tensorfold_b200 import _lib, synthetic
from tensorfold_b200.cuda.kernels import qmm

from gpu_util import DEV, to_dev

pytestmark = pytest.mark.gpu


def stand_in(folder):
    """A library with every entry point that launches nothing: they return 0, and ``tf_qmm_set`` what ``*during`` returns."""

    text = "long long (*during)(void);\n" + "".join(
        f"long long {name}() {{ return {'during()' if name == 'tf_qmm_set' else 65536 if name.endswith('_bytes') else 0}; }}\n"
        for name in _lib.SIGNATURES)
    (folder / "stand_in.c").write_text(text)
    subprocess.run(["gcc", "-w", "-shared", "-fPIC", "-o", str(folder / "stand_in.so"), str(folder / "stand_in.c")], check=True)
    return folder / "stand_in.so"


def test_a_launch_holds_its_scratch_area(tmp_path):
    """Another thread may drop every scratch area while a launch has given up the interpreter lock; the memory of the one in
    use must not reach a new tensor before the call is back."""

    q = qmm.pack(*to_dev(*synthetic.raw_weight(256, 1024, 4, 64, 1)), 64)
    x = synthetic.activations(4, 1024, 2).to(DEV)
    want = qmm.matmul(x, q, sk=2)
    area = qmm._set_scratch[x.device.index, _lib.stream_of(x)]
    held, size, taken = area.data_ptr(), area.numel(), []
    del area

    def during():
        qmm.reset_scratch()
        keep = [torch.empty((size,), dtype=torch.uint8, device=DEV) for _ in range(2 * qmm.SCRATCH_AREAS)]
        taken.extend(t.data_ptr() for t in keep)
        return 0

    path, callback = stand_in(tmp_path), ctypes.CFUNCTYPE(ctypes.c_longlong)(during)
    ctypes.c_void_p.in_dll(ctypes.CDLL(str(path)), "during").value = ctypes.cast(callback, ctypes.c_void_p).value
    native = _lib.native()
    native.bind(str(path), _lib.ensure_device)
    try:
        qmm.matmul(x, q, sk=2)
    finally:
        native.bind(str(_lib.LIB_PATH), _lib.ensure_device)
    assert taken and held not in taken
    assert torch.equal(qmm.matmul(x, q, sk=2), want)          # a new area, zeroed


@pytest.mark.parametrize("pdl", [False, True])
def test_a_capture_takes_many_slices_without_a_scratch_area(pdl):
    """More than eight K slices can pass through memory that the graph owns, so such a call needs no area made before."""

    q = qmm.pack(*to_dev(*synthetic.raw_weight(256, 1024, 4, 64, 3)), 64)
    x = synthetic.activations(4, 1024, 4).to(DEV)
    want = qmm.matmul(x, q, sk=12)
    torch.cuda.synchronize()
    qmm.reset_scratch()
    graph, out = torch.cuda.CUDAGraph(), torch.zeros_like(want)
    with torch.cuda.graph(graph):
        qmm.matmul(x, q, sk=12, out=out, pdl=pdl)
    graph.replay()
    assert torch.equal(out, want)


def test_an_outgrown_area_stays_with_its_graphs():
    """A graph captured with a stream's area is replayed after a larger set made the stream a new one: the first area's
    memory must not have become another tensor's."""

    qmm.reset_scratch()
    q = qmm.pack(*to_dev(*synthetic.raw_weight(256, 1024, 4, 64, 5)), 64)
    wide = qmm.pack(*to_dev(*synthetic.raw_weight(128 * 150, 1024, 4, 64, 6)), 64)
    x = synthetic.activations(4, 1024, 7).to(DEV)
    want, graph, stream = qmm.matmul(x, q, sk=4), torch.cuda.CUDAGraph(), torch.cuda.Stream()
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        qmm.matmul(x, q, sk=4, out=out)
    key = (x.device.index, stream.cuda_stream)
    held, size = qmm._set_scratch[key].data_ptr(), qmm._set_scratch[key].numel()
    with torch.cuda.stream(stream):
        qmm.matmul(x, wide, sk=16)                            # 150 blocks x 16 slices of 8 KB: more than an area holds
    torch.cuda.synchronize()
    others = [torch.full((size,), 255, dtype=torch.uint8, device=DEV) for _ in range(2 * qmm.SCRATCH_AREAS)]
    with torch.cuda.stream(stream):
        others += [torch.full((size,), 255, dtype=torch.uint8, device=DEV) for _ in range(2 * qmm.SCRATCH_AREAS)]
    assert held not in [t.data_ptr() for t in others]
    graph.replay()
    assert torch.equal(out, want)
    assert qmm._set_scratch[key].numel() >= 2 * size
    qmm.reset_scratch()


def test_an_area_is_clear_for_the_stream_that_gets_it():
    """The first call makes the areas of later streams too; a stream that does not wait for that call's queue must find its
    area zero.  Only the areas are looked at."""

    qmm.reset_scratch()
    torch.cuda.synchronize()
    dirty = [torch.full((qmm.SCRATCH_BYTES,), 255, dtype=torch.uint8, device=DEV) for _ in range(2 * qmm.SCRATCH_AREAS)]
    torch.cuda.synchronize()
    assert dirty[0].any()                                      # (loads the kernel)
    del dirty                                                  # their memory is what new areas get
    index, first, second = torch.cuda.current_device(), torch.cuda.current_stream(), torch.cuda.Stream()
    torch.cuda._sleep(200_000_000)                             # about a tenth of a second of queue on the first stream
    qmm._scratch_for(index, first.cuda_stream, 1)
    with torch.cuda.stream(second):
        assert not qmm._scratch_for(index, second.cuda_stream, 1).any()
    torch.cuda.synchronize()
    qmm.reset_scratch()


def test_host_memory_is_refused_unless_it_is_pinned():
    """An address that the device cannot reach must not get to a kernel, whichever operand brings it."""

    q = qmm.pack(*to_dev(*synthetic.raw_weight(256, 1024, 4, 64, 8)), 64)
    host = qmm.Q4(q.weight.cpu(), None, None, q.n, q.k, q.gs)
    for m in (4, 24):
        x, out = synthetic.activations(m, 1024, 9).to(DEV), torch.empty((m, 256), dtype=torch.bfloat16)
        calls = [lambda: qmm.matmul(x, host), lambda: qmm.prefill_matmul(x, host), lambda: qmm.matmul_act(x, host, act="relu2"),
                 lambda: qmm.matmul_act(x, host, act="relu2", prefill=True), lambda: qmm.matmul(x, q, out=out),
                 lambda: qmm.prefill_matmul(x, q, out=out), lambda: qmm.matmul_act(x, q, act="relu2", out=out),
                 lambda: qmm.matmul(x, q, qmm.group_sums(x).cpu()), lambda: qmm.matmul(x, q, sk=2, reduce=False, part=torch.empty(2 * m * 256))]
        for call in calls:
            with pytest.raises(ValueError):
                call()
        pinned, want = torch.empty((m, 256), dtype=torch.bfloat16, pin_memory=True), qmm.matmul(x, q)
        qmm.matmul(x, q, out=pinned)
        torch.cuda.synchronize()
        assert torch.equal(pinned, want.cpu())
