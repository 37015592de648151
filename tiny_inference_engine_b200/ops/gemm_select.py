"""Which matrix-product kernel runs for which operands, and with which tiling.

float32 has no reduced-precision matrix mode: few rows run on the CUDA cores, more as exact sums of bfloat16 terms
(csrc/gemm_f32_split.cu), with smaller errors than FFMAs.
bfloat16 runs on the tensor cores (tcgen05) whenever TMA can address the operands (K and the
row strides multiples of 8 elements, 16-byte aligned bases), else on the CUDA cores.
"""
from __future__ import annotations

import contextlib
import functools
import math
import os
import threading

import torch

from ..errors import TieError
from .library import call as _call, library as _library

NUM_SMS = 148


def tc_takes(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> bool:
    K = a.shape[1]
    return (a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and out.dtype in (torch.bfloat16, torch.float32)
            and K % 8 == 0 and a.stride(0) % 8 == 0 and w.stride(0) % 8 == 0
            and a.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


# Microseconds on one B200, fitted to a sweep of Qwen3-4B's and 8B's products at 160 to 2,048 tokens (8 % mean
# error): a k-block of a 128 x 128 or 128 x 256 tile, the prologue and epilogue of a wave of tiles, and writing
# and reading back a million float partial sums.
_US_K_BLOCK = {128: 0.225, 256: 0.356}
_US_WAVE = {128: 3.2, 256: 7.0}
_US_MEGA_PARTIAL = 0.68


def _plain_cost(M: int, N: int, k_blocks: int, bn: int, splits: int) -> float:
    """Estimated time of the plain tiling: the launcher gives every split NUM_SMS // splits CTAs, each of which
    walks its tiles in turn."""
    per = math.ceil(k_blocks / splits)
    real = math.ceil(k_blocks / per)
    tiles = math.ceil(M / 128) * math.ceil(N / bn)
    ctas = tiles if tiles * real <= NUM_SMS else max(1, NUM_SMS // real)
    waves = math.ceil(tiles / min(ctas, tiles))
    return waves * (per * _US_K_BLOCK[bn] + _US_WAVE[bn]) + (real * M * N / 1e6 * _US_MEGA_PARTIAL if real > 1 else 0.0)


@functools.lru_cache(maxsize=None)
def plan(M: int, N: int, K: int, split_many: bool = True) -> tuple[int, int, int]:
    """(transposed, tile width, splits) for out[M, N] = a[M, K] w[N, K]^T on one CTA per tile.

    Up to 128 tokens the weights take the 128-row side of the MMA and the tokens the narrow side
    (width = the smallest of 16, 32, 64, 128 that holds them): the product is bound by streaming the
    weights, and k is cut into splits so that every SM has a CTA pulling bytes. More tokens: 128-token
    row tiles against 128- or 256-wide weight tiles with k cut into up to four splits, whichever the
    cost estimate above puts first: what matters there is how many waves of tiles the SMs need.
    `split_many` False keeps k whole above 128 tokens (for a consumer that wants the finished product)."""
    k_blocks = math.ceil(K / 64)
    if M <= 128:
        bn = next(b for b in (16, 32, 64, 128) if b >= M)
        tiles = math.ceil(N / 128)
        splits = 1
        if bn <= 64 and tiles < 2 * NUM_SMS:
            # Two CTAs share an SM (the ring is about 100 KB): as many splits as keep all CTAs
            # resident at once, while a split keeps 4 k-blocks and the float partial sums
            # (written and read once) stay well below the weight bytes.
            splits = max(1, min(2 * NUM_SMS // tiles, k_blocks // 4, K // (8 * M)))
        elif bn == 128 and tiles < NUM_SMS:
            splits = max(1, min(NUM_SMS // tiles, k_blocks // 16))      # one CTA per SM at this width
        return 1, bn, splits
    if N <= 128:
        tiles = math.ceil(M / 128)
        bn = next(b for b in (16, 32, 64, 128) if b >= N)
        return 0, bn, max(1, min(NUM_SMS // tiles, k_blocks // 16)) if split_many else 1
    best = None
    for bn in (128, 256):
        for splits in range(1, 5 if split_many else 2):
            if splits > 1 and k_blocks // splits < 8:
                break
            cost = _plain_cost(M, N, k_blocks, bn, splits)
            if best is None or cost < best[0] - 1e-6:
                best = (cost, bn, splits)
    return 0, best[1], best[2]


_step = threading.local()


@contextlib.contextmanager
def step_scratch(ws):
    """While a step is issued by this thread: split products whose caller brings no memory leave their sums in the step's workspace."""
    before, _step.ws = getattr(_step, "ws", None), ws
    try:
        yield
    finally:
        _step.ws = before


def _scratch_for(numel: int, device) -> torch.Tensor:
    """Scratch for split products whose caller gave none: the step's own (captured graphs and repeated layers use its address again), or
    outside a step memory of the call's own stream. None of it is shared, so engines in several threads or streams do not meet in it."""
    ws = getattr(_step, "ws", None)
    if ws is not None:
        return ws.flat("gemm.partial", numel, torch.float32, 1 << 20)
    return torch.empty(numel, dtype=torch.float32, device=device)


@functools.lru_cache(maxsize=None)
def partial_capacity(max_rows: int, N: int, K: int, split_many: bool = True) -> int:
    """The most float partial sums a product of up to `max_rows` tokens with these weights leaves
    (splits x tokens x N over every token count): what its scratch buffer is sized for once."""
    most = 0
    for M in range(1, max_rows + 1):
        splits = plan(M, N, K, split_many)[2]
        if splits > 1:
            most = max(most, splits * M * N)
    return most


# Pairs of SMs (cta_group::2): from 65 tokens on; up to 64 the weights stream through two CTAs an SM (`plan`).
PAIR_FROM, PAIR_MIN_COLUMNS = 64, 256

_NO_PAIR = os.environ.get("TIE_NO_PAIR_GEMM") == "1"
_ops = None

PAIR_WIDTHS = (256, 224, 192, 160, 128, 96, 64)
# Microseconds on one B200, fitted to a sweep of 15 products of Qwen3's and the other designs' widths at 72 to 2,048 tokens, every
# tile width and up to eight splits (2,300 launches, 6 % error; the estimate's choice costs 0.5 % more than the best of each on
# average): a 64-deep k-block of a tile of 256 rows by `width` columns (2 cycles a column on the tensor cores from 192 columns on;
# narrower tiles wait for their operands, 66 bytes a cycle and SM from L2), a tile's own cost, the last tile's epilogue, a million
# float partial sums on their way out. _REDUCE_*: adding them up again, in the kernel that consumes them or in one of its own.
_PAIR_US_K_BLOCK = {64: 0.190, 96: 0.199, 128: 0.205, 160: 0.213, 192: 0.253, 224: 0.278, 256: 0.321}
_PAIR_US_LAUNCH, _PAIR_US_TILE, _PAIR_US_TAIL, _PAIR_US_MEGA_PARTIAL = 3.55, 0.92, 1.12, 0.367
# What the fit does not know of, seen in chains of launches with weights from memory: rows that the transposed side writes in 2-byte pieces (us a
# column of a tile, once; 8,192 x 2,048 at 192 tokens 13.9 us with tiles of 96 on that side, 13.1 with 128 on the other), and a gated unit of
# the plain side, which keeps a wave longer (24,576 x 4,096 at 320 tokens: estimated at 61 us, 69.1; one CTA a tile 65.0).
_PAIR_US_COLUMN_STORES, _PAIR_US_COLUMN_GATED = 0.0098, 0.008
_REDUCE_US_MEGA_CONSUMER, _REDUCE_US_MEGA, _REDUCE_US_LAUNCH = 0.35, 0.6, 2.2
# The same for one CTA a tile of 128 rows (`plan`), from the same sweep.
_SINGLE_US_K_BLOCK, _SINGLE_US_WAVE = {128: 0.237, 256: 0.414}, {128: 1.3, 256: 3.9}
_SINGLE_US_LAUNCH, _SINGLE_US_MEGA_PARTIAL = 3.5, 0.48
_pairs = None


def resident_pairs() -> int:
    """Pairs of SMs that hold the pair kernel at once: asked of the library once, 0 where there are none or TIE_NO_PAIR_GEMM=1 says not to use
    any (74 without a GPU, for planning)."""
    global _pairs
    if _pairs is None:
        if not torch.cuda.is_available():
            return NUM_SMS // 2
        _pairs = 0 if _NO_PAIR else int(_library().tie_gemm_tc2_pairs())
    return _pairs


def _reduce_cost(M: int, N: int, splits: int, consumer: bool) -> float:
    mega = splits * M * N / 1e6
    return 0.0 if splits == 1 else mega * _REDUCE_US_MEGA_CONSUMER if consumer else _REDUCE_US_LAUNCH + mega * _REDUCE_US_MEGA


def _pair_cost(M: int, N: int, K: int, pairs: int, transposed: int, bn: int, splits: int, gated: bool = False) -> float:
    """Estimated time of the pair kernel: its work items (tiles x splits) go round the pairs in waves."""
    rows, cols = (N, M) if transposed else (M, N)
    waves = math.ceil(math.ceil(rows / 256) * math.ceil(cols / bn) * splits / pairs)
    per = math.ceil(math.ceil(K / 64) / splits)
    out = _PAIR_US_TAIL * bn / 256 + (_PAIR_US_TAIL * bn / 256 + _PAIR_US_MEGA_PARTIAL * splits * M * N / 1e6 if splits > 1 else 0.0)
    if gated and not transposed:
        out += waves * bn * _PAIR_US_COLUMN_GATED
    elif transposed and not gated and splits == 1:
        out += bn * _PAIR_US_COLUMN_STORES
    # of two that come out alike the wider one: fewer bytes from L2, which counts once the power limit sets the clock
    return (_PAIR_US_LAUNCH + waves * (per * _PAIR_US_K_BLOCK[bn] + _PAIR_US_TILE) + out) * (1.0 + 1e-4 * (256 - bn))


def _single_cost(M: int, N: int, K: int, bn: int, splits: int) -> float:
    per = math.ceil(math.ceil(K / 64) / splits)
    real = math.ceil(math.ceil(K / 64) / per)
    tiles = math.ceil(M / 128) * math.ceil(N / bn)
    ctas = tiles if tiles * real <= NUM_SMS else max(1, NUM_SMS // real)
    waves = math.ceil(tiles / min(ctas, tiles))
    return _SINGLE_US_LAUNCH + waves * (per * _SINGLE_US_K_BLOCK[bn] + _SINGLE_US_WAVE[bn]) + (_SINGLE_US_MEGA_PARTIAL * real * M * N / 1e6 if real > 1 else 0.0)


@functools.lru_cache(maxsize=None)
def pair_plan(M: int, N: int, K: int, pairs: int, split: bool, consumer: bool = False, gated: bool = False) -> tuple | None:
    """(transposed, tile width, splits) of the pair kernel for out[M, N] = a[M, K] w^T, or None where `plan`'s one CTA a tile is
    as good: up to 64 tokens, few columns, and where its row tiles of 128 save more than pairs do (257 to 384 tokens); and without pairs.

    Up to 256 tokens the weights may fill the 256-row side of a tile and the tokens the other (`transposed`). With `split` k may be
    cut so that every pair has work; `consumer`: whoever reads the product adds the splits (else a kernel of its own does). `gated`: the
    epilogue forms a gated unit."""
    if M <= PAIR_FROM or N < PAIR_MIN_COLUMNS or pairs < 1:
        return None
    k_blocks, best = math.ceil(K / 64), None
    most = plan(M, N, K, split)[2] if split else 1        # as many sums as one CTA a tile would leave: what their buffers are made for
    for transposed in ((1, 0) if M <= 256 else (0,)):
        for bn in PAIR_WIDTHS:
            if transposed and (bn >= M + 32 or 2 * bn < M):
                continue
            tiles = math.ceil(N / 256) * math.ceil(M / bn) if transposed else math.ceil(M / 256) * math.ceil(N / bn)
            for splits in range(1, most + 1):
                if splits > 1 and (tiles * splits > pairs or k_blocks // splits < 6):
                    break
                if math.ceil(k_blocks / math.ceil(k_blocks / splits)) != splits:
                    continue
                cost = _pair_cost(M, N, K, pairs, transposed, bn, splits, gated) + _reduce_cost(M, N, splits, consumer)
                if best is None or cost < best[0] - 1e-9:
                    best = (cost, transposed, bn, splits)
    if M > 128:
        _, bn, splits = plan(M, N, K, split)
        if _single_cost(M, N, K, bn, splits) + _reduce_cost(M, N, splits, consumer) < best[0]:
            return None
    return best[1:]


def pair_width(M: int, N: int, K: int, pairs: int) -> int:
    """The tile width of the pair kernel with whole k and the tokens on the 256-row side; the widest on a tie."""
    return min(PAIR_WIDTHS, key=lambda bn: (_pair_cost(M, N, K, pairs, 0, bn, 1), -bn))


def _gated(epilogue) -> bool:
    """Whether an epilogue is that of a gated unit: the output is half as wide as the product, and k stays whole."""
    return int(epilogue) in (1, 2, 4, 5, 6)


def gated_splits(M: int, N: int, K: int, act: int) -> int:
    """Into how many parts a gated product's k is cut, the unit formed where the sums are added. In a step the kernels on either side
    overlap more with the split one, until its sums weigh more than that: up to 16 tokens a split pays from three parts on (decode steps of
    1 to 16 requests against whole k: 1 to 3 % for 12,288 x 2,048 with a clamped unit, 3 to 5 % for 3,072 and 6,144 x 1,024, 1 % for 10,240 x
    2,560; but 12,288 x 2,048 with the plain SiLU or ReLU, whose kernel leaves room for the next one, is 2 % slower at one request and even at
    eight), above from four and with long k (8,192 x 2,048 and longer ones; whole k 2 to 4 % faster for 12,288 x 2,048 with the SiLU
    at 32 and 64 requests, even or 1 % faster for the others)."""
    splits = plan(M, N, K)[2]
    pays = splits >= (3 if act > 2 or K >= 2560 else 4) if M <= 16 else splits >= 4 and K >= 2048
    return splits if M <= PAIR_FROM and pays else 1


class GatedUnit:
    """What a gated unit in a product's epilogue takes beside its code: the clamped unit's limit, slope and shift, the biases of
    the biased ones (float32 [N / 2]), and how many columns stand behind the unit's in the output's rows, a one and zeros."""

    def __init__(self, limit: float = 0.0, slope: float = 1.0, up_shift: float = 0.0, bias_gate=None, bias_up=None, ones: int = 0):
        self.biases = (bias_gate, bias_up)               # (their memory)
        self.ones = int(ones)
        self.args = (0 if bias_gate is None else bias_gate.data_ptr(), 0 if bias_up is None else bias_up.data_ptr(), float(limit), float(slope),
                     float(up_shift), self.ones)


_PLAIN_UNIT = GatedUnit()


def _entry(name: str, unit: GatedUnit, *args):
    """The launcher's call: with the unit's own arguments where it has some (`<name>_unit`, the stream behind them)."""
    return (name, *args) if unit is _PLAIN_UNIT else (name + "_unit", *args[:-1], *unit.args, args[-1])


def gemm_tc(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, transposed=None, bn=None, splits=None, scratch=None,
            silu=False, partial_scratch=None, deep=None, pair=None, checked: bool = False, unit: GatedUnit = _PLAIN_UNIT):
    """The tensor-core product; the tiling can be forced (tests). Returns `out`, or a SplitSum when
    `partial_scratch` is given and k is split."""
    global _ops
    if _ops is None:
        from . import SplitSum, _need, _stream, dtype_code      # once: this runs hundreds of times in an eager step
        _ops = (SplitSum, _need, _stream, dtype_code)
    SplitSum, _need, _stream, dtype_code = _ops
    M, K = a.shape
    N = w.shape[0]
    _need(w.shape[1] == K and out.shape == (M, N // 2 if _gated(silu) else N),
          f"gemm: shapes {tuple(a.shape)} x {tuple(w.shape)}^T -> {tuple(out.shape)}")
    _need(a.stride(1) == 1 and w.stride(1) == 1 and out.stride(1) == 1, "gemm: last axes must be contiguous")
    _need(checked or tc_takes(a, w, out),
          "gemm_tc: operands must be bfloat16 with K and row strides multiples of 8, 16-byte aligned")
    forced = not (transposed is None and bn is None and splits is None)
    p = None if forced or pair is False else pair_plan(M, N, K, resident_pairs(), not silu and K > 0, partial_scratch is not None, _gated(silu))
    if pair and p is None:
        p = (transposed or 0, bn or pair_width(M, N, K, resident_pairs()), splits or 1)
    if p is not None:
        t, bn, splits = p
        leave = splits > 1 and partial_scratch is not None
        if splits > 1:
            scratch = partial_scratch(splits * M * N) if leave else scratch if scratch is not None else _scratch_for(splits * M * N, a.device)
        _call(*_entry("tie_gemm_tc2", unit, dtype_code(out), a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), w.stride(0),
                      out.stride(0), int(silu), 0, 0, bn, t, splits, scratch.data_ptr() if splits > 1 else 0, 0 if leave else 1, _stream()))
        return SplitSum(scratch, _library().tie_gemm_tc_real_splits(K, splits), M, N) if leave else out
    t, b, s = plan(M, N, K)
    transposed = t if transposed is None else int(transposed)
    bn = b if bn is None else bn
    splits = s if splits is None else splits
    if _gated(silu):
        splits = 1
        if not transposed:
            bn = max(bn, 32)
    leave = splits > 1 and partial_scratch is not None and not silu
    if leave:
        scratch = partial_scratch(splits * M * N)
    elif splits > 1 and scratch is None:
        scratch = _scratch_for(splits * M * N, a.device)
    _call(*_entry("tie_gemm_tc", unit, dtype_code(out), a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, a.stride(0),
                  w.stride(0), out.stride(0), transposed, bn, splits, scratch.data_ptr() if splits > 1 else 0, int(silu),
                  0 if leave else 1, int(deep if deep is not None else (not transposed or bn >= 128)), 0, 0, _stream()))
    if leave:
        return SplitSum(scratch, _library().tie_gemm_tc_real_splits(K, splits), M, N)
    return out


def check_status() -> None:
    """After a synchronize: raises if a tensor-core kernel gave up a bounded wait."""
    code = _library().tie_kernel_status()
    if code:
        where = {1: "a matrix product's TMA producer waiting for a free stage", 2: "a matrix product's MMA issuer waiting "
                 "for operands", 3: "a matrix product's epilogue waiting for the accumulator",
                 4: "a CTA of a pair waiting for its partner before it frees its tensor memory",
                 11: "an attention kernel's TMA producer waiting for a free stage",
                 12: "an attention kernel waiting for keys and values"}.get(code, f"code {code}")
        if code == 13:
            raise TieError("decode attention was given fewer splits than a context needs; that sequence's output was not written")
        raise TieError(f"a kernel gave up after its wait limit ({where}); its output is invalid")


def gemm(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, partial_scratch=None):
    from . import gemm_simt
    if a.shape[0] == 0:
        return out
    if tc_takes(a, w, out):
        return gemm_tc(a, w, out, partial_scratch=partial_scratch, checked=True)
    gemm_simt(a, w, out)
    return out


def gemm_silu(a: torch.Tensor, w_blocks: torch.Tensor, out: torch.Tensor, act: int = 1, unit: GatedUnit = _PLAIN_UNIT) -> None:
    from . import _need
    _need(w_blocks.shape[0] % 32 == 0 and tc_takes(a, w_blocks, out),
          "gemm_silu: needs bfloat16 operands TMA can address and gate/up rows in blocks of 16")
    if a.shape[0] > 0:
        gemm_tc(a, w_blocks, out, silu=act, unit=unit)


class BoundGemm:
    """out = a . w^T for one weight matrix, checked once: what the parts call hundreds of times a step.

    The weight's address, sizes and kernel family are fixed when the part binds its tensors; a call looks up
    the tiling of its token count (computed once per count) and goes straight to the launcher. `a` and `out`
    come from the step's workspace: rows contiguous, 16-byte aligned, the compute dtype (the parts' contract);
    anything the tensor-core kernels do not take falls back to `gemm` with its full checks.

    A weight that the tensor-core kernels take is kept in k-blocks (`ops.pack_k_blocks`, with `pack`): `.w` is then
    [ceil(K / 64), rows, 64] and `packed_rows` its number of rows; `.rows(a, b)` gives the product with a slice of
    its rows (the q rows of a stacked q/k/v weight) over the same memory."""

    unit = _PLAIN_UNIT      # (an attribute of its own only where it says something: what a layer holds is looked through every step)

    def __init__(self, w: torch.Tensor, silu=False, split_many: bool = True, pack: bool = True, _slice=None, unit: GatedUnit | None = None):
        self.silu, self.split_many = int(silu), split_many      # 0: none, 3: the squared ReLU, else a gated unit
        if unit is not None:
            self.unit = unit
        self.gated = _gated(silu)
        if _slice is not None:              # rows [row0, row0 + N) of a packed weight
            parent, row0, n = _slice
            self.w, self.N, self.K, self.packed_rows, self.row0, self.fast = parent.w, n, parent.K, parent.packed_rows, row0, True
        else:
            self.N, self.K = w.shape
            self.fast = (w.dtype == torch.bfloat16 and w.stride(1) == 1 and self.K % 8 == 0 and w.stride(0) % 8 == 0
                         and w.data_ptr() % 16 == 0 and (not self.gated or self.N % 32 == 0))
            self.packed_rows = self.row0 = 0
            if pack and self.fast and w.is_cuda:
                from . import pack_k_blocks
                w = pack_k_blocks(w)
                self.packed_rows = self.N
            self.w = w
        self.w_ptr, self.ldw = self.w.data_ptr(), (64 if self.packed_rows else self.w.stride(0))
        self._plans: dict[int, tuple] = {}

    def rows(self, begin: int, end: int) -> "BoundGemm":
        """The product with rows begin..end-1 of this weight (no SiLU epilogue)."""
        if not 0 <= begin < end <= self.N:
            raise ValueError(f"rows {begin}..{end} of a weight of {self.N} rows")
        if self.packed_rows:
            return BoundGemm(None, False, self.split_many, _slice=(self, self.row0 + begin, end - begin))
        return BoundGemm(self.w[begin:end], False, self.split_many, pack=False)

    def row_major(self) -> torch.Tensor:
        """The weight as [N, K] (a copy if it is kept in k-blocks): for callers that need it the plain way."""
        if not self.packed_rows:
            return self.w
        from . import unpack_k_blocks
        return unpack_k_blocks(self.w, self.K)[self.row0:self.row0 + self.N]

    def _plan(self, M: int, consumer: bool):
        # up to 128 tokens k may be split for anyone, above for those who did not ask for the finished product
        pair = pair_plan(M, self.N, self.K, resident_pairs(), not self.silu and (self.split_many or M <= 128), consumer, self.gated)
        if pair is not None:
            t, bn, splits = pair
        else:
            t, bn, splits = plan(M, self.N, self.K, self.split_many)
        if self.gated:
            splits = gated_splits(M, self.N, self.K, self.silu) if pair is None else 1
            if not t:
                bn = max(bn, 32)
        real = _library().tie_gemm_tc_real_splits(self.K, splits) if splits > 1 else 1
        p = (pair is not None, t, bn, splits, int(not t or bn >= 128), real)
        self._plans[M, consumer] = p
        return p

    def __call__(self, a: torch.Tensor, out: torch.Tensor, partial_scratch=None):
        M = a.shape[0]
        if M == 0:
            return out
        if not (self.fast and a.dtype == torch.bfloat16 and a.stride(1) == 1 and a.stride(0) % 8 == 0 and a.data_ptr() % 16 == 0
                and out.stride(1) == 1 and a.shape[1] == self.K and out.shape[1] == (self.N // 2 if self.gated else self.N)
                and out.shape[0] == M and out.dtype in (torch.bfloat16, torch.float32)):
            w = self.row_major()
            if self.gated:
                gemm_silu(a, w, out, self.silu, self.unit)
                return out
            if self.silu:                   # the squared ReLU behind whichever product takes the operands
                from . import squared_relu
                gemm(a, w, out)
                squared_relu(out, out)
                return out
            return gemm(a, w, out, partial_scratch)
        global _ops
        if _ops is None:
            from . import SplitSum, _need, _stream, dtype_code
            _ops = (SplitSum, _need, _stream, dtype_code)
        SplitSum, _, _stream, dtype_code = _ops
        consumer = partial_scratch is not None and not self.silu
        pair, t, bn, splits, deep, real = self._plans.get((M, consumer)) or self._plan(M, consumer)
        code = 1 if out.dtype == torch.bfloat16 else 0
        leave = splits > 1 and consumer
        scratch = 0
        if leave:
            buf = partial_scratch(splits * M * self.N)
            scratch = buf.data_ptr()
        elif splits > 1:        # added up here: a gated unit's caller brings memory of its own step
            n = splits * M * self.N
            buf = partial_scratch(n) if partial_scratch is not None else _scratch_for(n, a.device)
            scratch = buf.data_ptr()
        if pair:
            args = (code, a.data_ptr(), self.w_ptr, out.data_ptr(), M, self.N, self.K, a.stride(0), self.ldw, out.stride(0), self.silu,
                    self.packed_rows, self.row0, bn, t, splits, scratch, 0 if leave else 1)
        else:
            args = (code, a.data_ptr(), self.w_ptr, out.data_ptr(), M, self.N, self.K, a.stride(0), self.ldw, out.stride(0),
                    t, bn, splits, scratch, self.silu, 0 if leave else 1, deep, self.packed_rows, self.row0)
        name = "tie_gemm_tc2" if pair else "tie_gemm_tc"
        if self.unit is _PLAIN_UNIT:
            _call(name, *args, _stream())
        else:
            _call(name + "_unit", *args, *self.unit.args, _stream())
        if leave:
            return SplitSum(buf, real, M, self.N)
        return out
