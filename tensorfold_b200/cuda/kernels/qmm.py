"""4-bit lane matmul: rows run the same groups and K slices at any row count, so no row affects another.

Host-side mirror of the reference module ``tensorfold.cuda.kernels.qmm`` (cuda/kernels/qmm.py:24-171): same names,
argument meaning and errors; the arithmetic runs in ``libtensorfold_b200.so``.
"""

from __future__ import annotations

import os
from dataclasses import dataclass
from functools import lru_cache

import torch

from ... import _lib

BITS = (2, 3, 4, 5, 6, 8)
GROUPS = (32, 64, 128)


@lru_cache(maxsize=1)
def _native():
    """The extension module, told the two rules that stay here: K slices of a shape, and a stream's scratch."""

    module = _lib.native()
    module.hooks(default_split, _scratch_for)
    return module


@lru_cache(maxsize=None)
def _unit_words(bits: int, gs: int) -> int:
    return _lib.lib().tf_unit_words(bits, gs)


@dataclass
class Q4:
    """A packed (n, k) weight in the tiled layout: int32 units [ceil(n / 128), k / gs, unit words], each unit the codes
    of 128 output columns for one group followed by their 128 (scale, bias) bf16 pairs.  ``scales`` and ``biases`` stay
    None: the pairs live inside ``weight`` (``unpack`` returns them).  Field order follows cuda/kernels/qmm.py:24-35."""

    weight: torch.Tensor
    scales: torch.Tensor | None
    biases: torch.Tensor | None
    n: int
    k: int
    gs: int
    bits: int = 4

    def nbytes(self) -> int:
        return self.weight.numel() * self.weight.element_size()


def pack(weight: torch.Tensor, scales: torch.Tensor, biases: torch.Tensor, gs: int, chunk: int = 4096,
         bits: int = 4) -> Q4:
    """MLX (n, k * bits / 32) words, (n, k / gs) bf16 scales and biases -> ``Q4``.  ``chunk`` is accepted for
    signature parity (cuda/kernels/qmm.py:55) and unused: the repack is one kernel."""

    if bits not in BITS or gs not in GROUPS:
        raise ValueError("affine weights require 2/3/4/5/6/8 bits and groups of 32/64/128")
    if weight.dim() != 2 or weight.dtype not in (torch.int32, torch.uint32):
        raise ValueError("pack: weight must be 2-D int32/uint32 MLX words")
    if scales.dtype != torch.bfloat16 or biases.dtype != torch.bfloat16 or scales.shape != biases.shape:
        raise ValueError("pack: scales and biases must be matching bf16 tensors")
    n, words = weight.shape
    k = words * 32 // bits
    if scales.shape != (n, k // gs) or k % gs or (k * bits) % 32:
        raise ValueError(f"pack: words {tuple(weight.shape)} do not match scales {tuple(scales.shape)} at {bits} bits")
    stream = _lib.stream_of(weight)
    weight, scales, biases = weight.contiguous(), scales.contiguous(), biases.contiguous()
    out = torch.empty((-(-n // 128), k // gs, _unit_words(bits, gs)), dtype=torch.int32, device=weight.device)
    _native().tf_pack("pack", weight, scales, biases, n, k, bits, gs, out, stream)
    return Q4(out, None, None, n, k, gs, bits)


def unpack(q: Q4, chunk: int = 64) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """The stored MLX layout again: (n, k * bits / 32) int32 words, (n, k / gs) bf16 scales and biases."""

    stream = _lib.stream_of(q.weight)
    dev = q.weight.device
    words = torch.empty((q.n, q.k * q.bits // 32), dtype=torch.int32, device=dev)
    scales = torch.empty((q.n, q.k // q.gs), dtype=torch.bfloat16, device=dev)
    biases = torch.empty_like(scales)
    tiled = q.weight if q.weight.is_contiguous() else q.weight.contiguous()
    _native().tf_unpack("unpack", tiled, q.n, q.k, q.bits, q.gs, words, scales, biases, stream)
    return words, scales, biases


def split_k(n: int, k: int, gs: int = 64, target: int = 192) -> int:
    """K slices for an (n, k) weight: a function of the shape only (never of the row count)."""

    tiles, groups, sk = -(-n // 64), k // gs, 1
    while sk < 8 and tiles * sk < target and groups % (sk * 2) == 0 and groups // (sk * 2) >= 8:
        sk *= 2
    return sk


LANES = 592            # 128-column lanes the persistent decode kernel streams side by side on a B200: 148 SMs x 4
MIN_GROUPS = 6         # groups a K slice should hold at least (three pipeline stages of 128 inputs at groups of 64)


def default_split(n: int, k: int, gs: int = 64, share: float = 1.0) -> int:
    """The K slices ``matmul`` uses when it is given none: a function of the shape only (never of the row count), chosen
    so that the projection's (128-column block, slice) units fill the machine's lanes once: LANES / blocks, at least
    MIN_GROUPS groups a slice.  Slices need not divide the groups evenly (slice s covers groups
    [s G / sk, (s + 1) G / sk)).  ``share`` is for projections an engine always launches as a set (q/k/v, gate/up):
    the set's 128-column blocks over this projection's, so that the SET fills the lanes once (2 for gate or up)."""

    blocks, groups = -(-n // 128), k // gs
    sk = int(LANES // max(1.0, blocks * share))
    return max(1, min(sk, groups // MIN_GROUPS if groups >= MIN_GROUPS else 1))


def set_splits(shapes, gs: int = 64) -> list[int]:
    """K slices for projections an engine always launches together (``matmul_set``): [(n, k), ...] -> one slice count
    each, so that the set's units fill the lanes once.  A load-time decision, like stacking: a projection's bits depend
    on its slice count, so it must use the same count wherever it runs."""

    blocks = [-(-n // 128) for n, _ in shapes]
    return [default_split(n, k, gs, share=sum(blocks) / b) for (n, k), b in zip(shapes, blocks)]


def bucket(m: int) -> int:
    """The reference's row tile (16, 32, else 64); kept for callers that size buffers by it.  Tiles never change bits."""

    if m < 1:
        raise ValueError("the lane matmul takes at least one row")
    return 16 if m <= 16 else 32 if m <= 32 else 64


def group_sums(x: torch.Tensor, gs: int = 64) -> torch.Tensor:
    """(M, K) bf16 (rows may be strided) -> (M, K/gs) fp32 sums of each group's inputs, with the matmul's own bits."""

    if x.dtype != torch.bfloat16 or x.dim() != 2 or x.shape[1] % gs:
        raise ValueError("group_sums: x must be (M, K) bf16 with K a multiple of the group")
    if x.stride(1) != 1 or (x.shape[0] > 1 and x.stride(0) % 2) or x.data_ptr() % 4:
        x = x.clone(memory_format=torch.contiguous_format)
    stream = _lib.stream_of(x)
    m, k = x.shape
    xs = torch.empty((m, k // gs), dtype=torch.float32, device=x.device)
    _native().tf_group_sums("group_sums", x, x.stride(0), m, k, gs, xs, stream)
    return xs


def matmul(x: torch.Tensor, q: Q4, xs: torch.Tensor | None = None, *, sk: int | None = None, f32: bool = False,
           out: torch.Tensor | None = None, part: torch.Tensor | None = None, reduce: bool = True,
           pdl: bool = False) -> torch.Tensor:
    """x @ q.T as (M, n) bf16, or unrounded fp32 with ``f32``; ``reduce=False`` returns K slices to add in order.

    ``pdl`` (not in the reference) launches with programmatic stream serialisation so the weight prefetch of this call
    overlaps the end of the previous kernel in the stream: the weights must not be what a kernel still in flight writes."""

    return _native().matmul(x, q, xs, sk, f32, out, part, reduce, pdl, STREAM)


STREAM = os.environ.get("TENSORFOLD_B200_STREAM", "1") != "0"      # decode windows run the persistent kernel (same bits)
SCRATCH_BYTES = 16 << 20          # one scratch area: room for a gate/up set of 17408 rows each in 4 K slices
SCRATCH_AREAS = 4                 # areas made on a device's first call: the calling stream's and three side streams'
_set_scratch: dict = {}           # (device index, stream) -> the stream's scratch area
_free_areas: dict = {}            # device index -> areas not yet handed to a stream
_outgrown: list = []              # areas that were too small for a later call: graphs captured with them may still be replayed


def _scratch_for(index: int, stream: int, need: int) -> torch.Tensor:
    """The scratch area of (device index, stream) where the K slices of a set meet: zeroed once, left zero by every call.
    The extension asks for it when it has not seen the stream, or the area it knows is too small.

    Areas are made eagerly (four on a device's first call, more when a fifth stream shows up or a set needs more room)
    and only handed out during a stream capture: a graph must not own memory that later calls use, so a capture that
    would need a new allocation is refused with a message saying which eager call to make first.  An area that a stream
    outgrows is kept for graphs; a new one is at least twice its size, so all of those are smaller than the last."""

    device, key = torch.device("cuda", index), (index, stream)
    buf = _set_scratch.get(key)
    if buf is not None and buf.numel() >= need:
        return buf
    capturing = torch.cuda.is_current_stream_capturing()
    free = _free_areas.setdefault(index, [])
    if not free and not capturing and not any(k[0] == index for k in _set_scratch):
        maker = torch.cuda.Stream(device=device)                # cleared for every stream, not only after this one's queue
        with torch.cuda.stream(maker):
            free.extend(torch.zeros((SCRATCH_BYTES,), dtype=torch.uint8, device=device) for _ in range(SCRATCH_AREAS))
        maker.synchronize()
    fits = [i for i, area in enumerate(free) if area.numel() >= need]
    if buf is None and fits:
        buf = free.pop(fits[0])
        buf.record_stream(torch.cuda.current_stream(device))    # freed, its memory waits for the work queued here
    elif capturing:
        raise RuntimeError("matmul_set: this call needs a new scratch area, which cannot be made while the stream is "
                           "capturing; run it once eagerly (any stream of this device) before the capture")
    else:
        size = max(need, SCRATCH_BYTES)
        if buf is not None:
            _outgrown.append(buf)
            size = max(size, 2 * buf.numel())
        buf = torch.zeros((size,), dtype=torch.uint8, device=device)
    _set_scratch[key] = buf
    return buf


def reset_scratch() -> None:
    """Forget every scratch area (after ``device_error`` reported a lost wait their counters may be non-zero).  Graphs
    captured before must not be replayed after it: they use the areas of their time."""

    _set_scratch.clear()
    _free_areas.clear()
    _outgrown.clear()
    _native().forget_scratch()


def matmul_set(x: torch.Tensor, qs, xs: torch.Tensor | None = None, *, sks=None, f32: bool = False, outs=None,
               pdl: bool = False) -> list:
    """Several projections of the SAME rows (q/k/v, gate/up) in one persistent launch: [x @ q.T for q in qs], each with
    the bits ``matmul(x, q, sk=sk)`` gives.  1 to 16 rows, up to 4 weights of one format and K.  Not in the reference,
    whose engines issue these as separate calls (families/qwen3_5/cuda/qmm_fast.py:49-64)."""

    return _native().matmul_set(x, qs, xs, sks, f32, outs, pdl)


def prefill_matmul(x: torch.Tensor, q: Q4, *, f32: bool = False, tile: int = 0,
                   out: torch.Tensor | None = None) -> torch.Tensor:
    """Prefill: weights rounded once to bf16, one fp32 chain over K on the tcgen05 tensor cores; any chunking gives the
    same bits, not decode's.  ``tile`` is accepted for signature parity (cuda/kernels/qmm.py:160) and unused.  Formats
    the tcgen05 kernel does not take (other widths, groups of 128, K not a multiple of 64) run through ``matmul``."""

    if q.bits != 4 or q.gs not in (32, 64) or q.k % 64:
        return matmul(x, q, f32=f32, out=out)
    return _native().prefill_matmul(x, q, f32, out)


_side_streams: dict = {}


def fork_join(calls) -> None:
    """Runs independent launches side by side: ``calls`` are thunks that launch on the current stream (projections that
    read the same input, like q/k/v or gate/up).  The first runs on the current stream, the others on side streams that
    wait for everything already queued on it; the current stream then waits for all of them.  Works eagerly and under
    CUDA-graph capture (the waits become graph edges).  A decode-sized projection cannot fill the GPU on its own (its
    launch, first-byte latency and slice reduction are fixed costs), so independent ones overlap nearly for free.

    Tensors a thunk allocates belong to its side stream's pool: give the thunks preallocated outputs (``out=``) for
    anything the main stream reads after the join, or call ``record_stream(main)`` on what they return; a tensor made
    and consumed inside one thunk needs neither."""

    calls = list(calls)
    if len(calls) < 2:
        for fn in calls:
            fn()
        return
    main = torch.cuda.current_stream()
    pool = _side_streams.setdefault(main.device, [])
    while len(pool) < len(calls) - 1:
        pool.append(torch.cuda.Stream(device=main.device))
    fork = torch.cuda.Event()
    fork.record(main)
    calls[0]()
    for fn, side in zip(calls[1:], pool):
        side.wait_event(fork)
        with torch.cuda.stream(side):
            fn()
        done = torch.cuda.Event()
        done.record(side)
        main.wait_event(done)


def pack_pair(gate: tuple, up: tuple, gs: int, bits: int = 4) -> Q4:
    """Gate and up projections (each MLX words, scales, biases of n rows) as ONE weight of 2 n rows that interleaves 16
    gate rows with 16 up rows, so a matmul tile pair holds both halves of every SwiGLU output (see ``matmul_act``)."""

    (wg, sg, bg), (wu, su, bu) = gate, up
    if wg.shape != wu.shape or sg.shape != su.shape or wg.dim() != 2:
        raise ValueError("pack_pair: gate and up must have the same 2-D shapes")
    n, words = wg.shape
    k = words * 32 // bits
    if n % 16 or k % gs or any(t.dtype != torch.bfloat16 for t in (sg, bg, su, bu)):
        raise ValueError("pack_pair: rows in whole 16-row tiles, bf16 scales and biases")
    stream = _lib.stream_of(wg)
    ts = [t.contiguous() for t in (wg, sg, bg, wu, su, bu)]
    out = torch.empty((-(-2 * n // 128), k // gs, _unit_words(bits, gs)), dtype=torch.int32, device=wg.device)
    _native().tf_pack_pair("pack_pair", *ts, n, k, bits, gs, out, stream)
    return Q4(out, None, None, 2 * n, k, gs, bits)


def matmul_act(x: torch.Tensor, q: Q4, *, act: str = "swiglu", limit: float = 0.0, out: torch.Tensor | None = None,
               pdl: bool = False, prefill: bool = False) -> torch.Tensor:
    """Projection with the experts' activation epilogue, dense form: ``act="swiglu"`` on a ``pack_pair`` weight gives
    bf16(bf16(silu(bf16 gate)) * bf16 up) as (M, n / 2); ``act="relu2"`` gives bf16(relu(bf16 v)^2) as (M, n)."""

    if act not in ("swiglu", "relu2"):
        raise ValueError("matmul_act: act is 'swiglu' or 'relu2'")
    return _native().matmul_act(x, q, act == "swiglu", limit, out, pdl, prefill)
