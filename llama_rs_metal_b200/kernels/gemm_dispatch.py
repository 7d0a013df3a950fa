"""Which bfloat16 matrix-product kernel runs for a shape.

* up to 64 rows (decode steps): tcgen05 with the weights as its wide operand (csrc/gemm_bf16_few.cu),
  in K slices where the product is narrow and its reader adds planes; few_plan says where it is the
  faster one;
* up to 8 rows of smaller matrices, and what is narrow and cannot be cut: the weight-streaming kernel
  (csrc/gemm_bf16_stream.cu);
* more than 64 rows, wherever its tiles are estimated to waste less (no fixed number of rows): tcgen05
  over pairs of SMs with the weights as the wide operand (csrc/gemm_bf16_wide.cu; wide_plan);
* else (prompts): the TMA + tcgen05 kernel
  (csrc/gemm_bf16_umma.cu), with 128 x 128, 128 x 256 or 256 x 256 tiles, whichever needs less
  time by a count of rounds over the SMs and the measured cost of a tile;
* a narrow product that is to be added to the residual stream may be cut into K slices so that
  every SM works: the slices are stored as planes of an [slices, M, N] tensor, which the next
  norm adds in slice order (gemm_bf16_slices); nothing meets by atomics, so the same step gives
  the same bits every time;
* every shape the others refuse (K not a multiple of 8, unaligned views): the
  warp-level tiled kernel (csrc/gemm_bf16_mma.cu), which takes any M, N, K.
"""
from __future__ import annotations

import ctypes
import functools
from typing import Dict, Optional

import torch

from ..errors import LlamaError
from . import library
from .ops import _done, _ptr, _stream  # noqa: PLC2701  (same package)

SM_COUNT = 148
force_tiled = False  # tests switch the fast kernels off to compare both paths
no_wide = False  # tests: products of more than 64 rows stay off the kernel with the weights as the wide operand
wide_shape = None  # tests and tuning: (activation rows of a tile, K slices) of that kernel instead of its own rule
umma_width: Optional[int] = None  # tests pin the tile: 128 (128 x 128), 256 (128 x 256), 512 (256 x 256), 192 (128 x 192)

_status: Dict[int, torch.Tensor] = {}
_status_dirty = False
_status_launches = 0  # launches (or captures) so far of kernels that write the status word


def mark_status_dirty() -> None:
    """A kernel with bounded waits was launched (directly, or by replaying a CUDA graph that holds
    one): the next check_status() reads the status word."""
    global _status_dirty, _status_launches
    _status_dirty = True
    _status_launches += 1


def status_launch_count() -> int:
    return _status_launches


def _status_word(device: torch.device) -> torch.Tensor:
    index = device.index if device.index is not None else torch.cuda.current_device()
    if index not in _status:
        _status[index] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[index]


def check_status() -> None:
    """Raise if a tensor-core kernel gave up on a wait since the last check (reads 4 bytes back)."""
    global _status_dirty
    if not _status_dirty:
        return
    _status_dirty = False
    for word in _status.values():
        code = int(word.item())
        if code != 0:
            word.zero_()
            names = {1: "a free stage", 2: "operand tiles", 3: "the accumulator", 4: "copies in flight",
                     5: "a free accumulator", 21: "the query tiles", 22: "a key/value tile", 23: "scores",
                     24: "probabilities", 25: "the output", 26: "a free key/value stage", 27: "aligned shared memory"}
            names.update({31: "a free stage", 32: "operand tiles", 33: "the accumulator", 34: "copies in flight",
                          35: "a free accumulator"})
            names.update({41: "the query tile", 42: "a key/value tile", 43: "scores", 44: "probabilities", 45: "the output",
                          46: "a free key/value stage", 47: "aligned shared memory"})
            names.update({51: "a free stage", 52: "operand tiles", 53: "the accumulator", 54: "copies in flight",
                          55: "a free accumulator"})
            names.update({61: "a free stage", 62: "operand parts", 63: "the accumulator", 64: "operand tiles", 65: "copies in flight",
                          66: "a free tile", 67: "the small products"})
            names.update({71: "a free stage", 72: "operand tiles", 73: "the accumulator", 74: "copies in flight", 75: "a free accumulator",
                          76: "gates and ups"})
            kernel = "gemm_bf16_wide" if code >= 71 else "gemm_f32_umma" if code >= 61 else "gemm_bf16_few" if code >= 51 else "attention_gated_umma" if code >= 41 else "gemm_bf16_umma_pair" \
                if code >= 31 else "attention_prefill_pingpong" if code >= 21 else "gemm_bf16_umma"
            raise LlamaError(f"{kernel} gave up waiting for {names.get(code, code)}; its result is invalid")


# What an output tile costs relative to a 128 x 128 one. Operand traffic from L2 bounds these
# products (measured: the tensor pipe is busy 38-44 % of the time with 128 x 128 tiles, 66-71 %
# with 128 x 256), so a larger tile does more work per byte. A 256 x 256 tile fills the tensor
# memory, so its epilogue does not run under the next tile's MMAs: it pays only when K is long
# (measured at 8,192 rows: 0.85 of the 128 x 256 time at K = 8192, 1.05 at K = 2048 with a plain
# epilogue, 1.3 with the SiLU gate).
def _tile_costs(K: int, mode: int):
    k_blocks = max(1, -(-K // 64))
    epilogue = 1.1 if mode == 3 else 0.55
    return ((128, 128, 1.0), (128, 256, 1.4), (256, 256, 1.4 * (1.55 + epilogue * 32 / k_blocks)), (128, 192, 1.2))


PAIR = 4  # tile code of the kernel that runs a 256 x 256 tile on two SMs


def _pair_cost(K: int, rounds: int) -> float:
    """`rounds` rounds of 256 x 256 tiles over the pairs of SMs, in units of a 128 x 128 tile on one
    SM: each SM does a 128 x 256 tile's work with a third less operand traffic and a hidden
    epilogue (measured at 2,048 rows: gate/up 104 us against 115, down 60 against 64, the 8B shape's
    QKV 88 against 97; at 4,096 rows 5-15 % faster than the best single-SM tile throughout); its
    start-up (a cluster to place, tensor memory allocated by both CTAs together) weighs more the
    shorter K is."""
    return 1.27 * rounds + 0.2 * 32 / max(1, -(-K // 64))


_pair_room = {}


def pair_room() -> int:
    """Pairs of SMs the two-CTA product can occupy at once (0: not on this device)."""
    device = torch.cuda.current_device()
    if device not in _pair_room:
        _pair_room[device] = 0 if force_tiled else int(library.load().lrm_gemm_bf16_umma_pair_room())
    return _pair_room[device]


def tile_choice(M: int, N: int, K: int = 2048, mode: int = 0, pairs: int = 0, multiple_of: int = 1) -> int:
    """0: 128 x 128, 1: 128 x 256, 2: 256 x 256, 3: 128 x 192 output tiles on one SM each, or 4: 256 x
    256 tiles on `pairs` pairs of SMs (0: not to be had): least rounds over the SMs times cost, among
    the tiles whose width is a multiple of `multiple_of` (an epilogue that works on whole heads)."""
    if umma_width is not None and {128: 128, 256: 256, 512: 256, 192: 192, "pair": 256}[umma_width] % multiple_of == 0:
        return {128: 0, 256: 1, 512: 2, 192: 3, "pair": PAIR}[umma_width]
    best, best_cost = 0, None
    for index, (rows, columns, cost) in enumerate(_tile_costs(K, mode)):
        if columns % multiple_of or (pairs > 0 and index == 2):  # a pair does what the 256 x 256 tile does, better
            continue
        rounds = -(-(-(-M // rows) * -(-N // columns)) // SM_COUNT)
        if best_cost is None or rounds * cost < best_cost:
            best, best_cost = index, rounds * cost
    if pairs > 0 and mode <= 3:
        rounds = -(-(-(-M // 256) * -(-N // 256)) // pairs)
        if _pair_cost(K, rounds) < best_cost:
            best = PAIR
    return best


def _tile_time(M: int, N: int, K: int, mode: int, pairs: int) -> float:
    """us that tile_choice's tile is estimated to take, on the scale of wide_plan: 0.3 us for 64 of K of a 128 x 128 tile."""
    k_blocks = -(-K // 64)
    costs = [-(-(-(-M // rows) * -(-N // columns)) // SM_COUNT) * cost for index, (rows, columns, cost) in enumerate(_tile_costs(K, mode))
             if not (pairs > 0 and index == 2)]
    if pairs > 0:
        costs.append(_pair_cost(K, -(-(-(-M // 256) * -(-N // 256)) // pairs)))
    return max(min(costs) * k_blocks * 0.3, N * K * 2 / 6e6) + 4.0


# us for 64 of K of a tile of 256 weight rows and so many activation rows on a pair of SMs
WIDE_BLOCK = {64: 0.21, 96: 0.215, 128: 0.23, 160: 0.265, 192: 0.29, 224: 0.345, 256: 0.40}


@functools.lru_cache(maxsize=4096)
def wide_plan(M: int, N: int, K: int, mode: int, pairs: int):
    """(activation rows of a tile, K slices) on the kernel with the weights as the wide operand, or None where the other tiles are
    estimated to be faster. Mode 2 may be cut into K slices, whose planes the next norm adds; the others never are.

    An item's time is its blocks of 64 of K times WIDE_BLOCK, as measured in steady state (389 cycles at 192 rows, whose products take
    384; the clock falls with the width under the power cap), 5 us a product for start-up and the last epilogue, and the weights come
    at 6.2 TB/s at best. A plane costs its write and the norm's read. us, in brackets the tiles with the activations as the wide operand, in
    chains over more weights than L2 holds: 3072 x 2048 128 rows 9.2 (12.1), 529 rows 11.5 (12.2); 6144 x 4096 128 rows 16.7 (21.1), 529 rows
    23.4 (27.4), 1,024 rows 40.6 (44.7); gated 16384 x 2048 180 rows 17.2 (20.0), 529 rows 32.0 (37.8); gated 28672 x 4096 300 rows 72.5
    (84.9), 529 rows 99.8 (115.9); 2048 x 2048 529 rows 10.4 (13.0), 2,500 rows 20.0 (26.0); 4096 x 14336 300 rows 35.0 in two planes
    (41.4 in three), 600 rows 61.2 (74.6), 1,280 rows 121 (171). Where full tiles of 256 x 256 on the pairs fill their rounds they are as
    good or better: gated 28672 x 4096 1,024 rows 169 against 180, 4096 x 14336 2,048 rows 170 against 173."""
    best = _wide_best(M, N, K, 8 if mode == 2 else 1, pairs)
    sliced = mode == 2 and best[2] > 1
    if not sliced and 0.97 * _tile_time(M, N, K, mode, pairs) <= best[0]:
        return None
    return best[1], best[2]


def _wide_best(M: int, N: int, K: int, most: int, pairs: int):
    """(us, activation rows of a tile, K slices, at most `most`) of the best tiles there by wide_plan's estimate."""
    k_blocks, columns = -(-K // 64), -(-N // 256)
    best = None
    for rows, block in WIDE_BLOCK.items():
        tiles = columns * -(-M // rows)
        for wanted in range(1, most + 1):
            per_slice = -(-k_blocks // wanted)
            slices = -(-k_blocks // per_slice)
            if slices != wanted or (slices > 1 and per_slice < 4):
                continue
            time = max(-(-tiles * slices // pairs) * per_slice * block, N * K * 2 / 6.2e6) + 5.0
            if slices > 1:
                time += slices * (2.0 * M * N * 4 / 3.5e6)
            if best is None or time < best[0]:
                best = (time, rows, slices)
    return best


@functools.lru_cache(maxsize=4096)
def cut_plan(M: int, N: int, K: int, pairs: int) -> bool:
    """Whether a product whose float32 result is wanted at once (no norm behind it adds planes) is cut into K slices all the same, the
    planes of few_plan or wide_plan, with a launch that adds them up: where a long K leaves most SMs idle or one after another.

    us, whole and cut with the addition, weights from memory: up to 64 rows, 2048 x 8192 16 rows 16 and 10, 64 rows 40 and 11; 4096 x 14336 8
    rows 24 and 23, 16 rows 32 and 24, 64 rows 76 and 27; 1024 x 4096 16 rows 7 and 6, 64 rows 17 and 8; 3072 x 2048 32 rows 9 and 6; under the
    line 2048 x 2048 16 rows 5 and 6, 4096 x 8192 8 rows 14 and 15, 8192 x 2048 48 rows 13 and 14. More rows, by wide_plan's estimate and 3 us for
    the launch: 2048 x 8192 100 rows 27 and 14, 500 rows 29 and 25; 4096 x 14336 100 rows 45 and 30, 300 rows 48 and 40; under the line 2048 x 2048 300
    rows 10 and 12, 6144 x 4096 100 rows 17 and 18."""
    if M > 64:
        best = _wide_best(M, N, K, 8, pairs)
        return best[2] > 1 and best[0] + 3.0 < min(_wide_best(M, N, K, 1, pairs)[0], _tile_time(M, N, K, 2, pairs))
    if M <= STREAM_ROWS:
        return N * K >= 40e6
    if M <= 16:
        return K >= 6144
    return K >= (4096 if M <= 32 and N < 3072 else 2048) and (K > 2048 or N < 8192)


def _wide(x: torch.Tensor, weight: torch.Tensor, mode: int, umma_ok: bool):
    """wide_plan where that kernel takes the product at all."""
    M, K = x.shape
    N = weight.shape[0]
    if M <= 64 or not umma_ok or no_wide or umma_width is not None or N % 2 or (mode == 3 and N % 16):
        return None
    pairs = pair_room()
    if pairs == 0:
        return None
    return wide_shape or wide_plan(M, N, K, mode, pairs)


def sorted_on_pairs() -> bool:
    """Whether a prompt's sorted experts go through pairs of SMs with the weights as the wide operand: wherever those are to be had. us
    over router and experts, in brackets 128 x 256 tiles of one SM each, before the passes around them became shorter: 2048 x 1024, 2 of
    8 experts 1,500 tokens 82.7 (87.4), 2,048 103 (117), 4 of 16 1,000 tokens 120 (123); 1024 x 512 2 of 8 520 tokens 31.8 (34.8), 2,000 54.2
    (60.9)."""
    return not (no_wide or no_fused_gate) and umma_width is None and pair_room() > 0


def gemm_bf16_wide(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, mode: int, rows: int, slices: int = 1) -> None:
    """gemm_bf16 (modes 0 to 3), or K slices as planes [slices, M, N] (mode 4), in tiles of 256 weight rows and `rows` rows of x."""
    M, K = x.shape
    mark_status_dirty()
    _done(library.load().lrm_gemm_bf16_wide(_ptr(x), _ptr(weight), _ptr(out), M, weight.shape[0], K, mode, rows, slices,
                                            _ptr(_status_word(x.device)), _stream()), "gemm_bf16_wide")


STREAM_ROWS = 8  # up to this many rows the streaming kernel is faster than the tiles with the rows as the wide operand
force_stream = False  # tests: keep 17-64 rows on the streaming kernel
stream_shape = None  # tests and tuning: (warps per CTA, K slices) of the streaming kernel instead of its own rule


def _few_rows_plan(M: int, N: int, K: int, mode: int):
    """For 9-64 rows: (use the tensor-core kernel?, K slices). Measured at the 1B layer sizes:
    many column tiles run as they are from 13 rows on; a product whose slices the next norm adds
    (mode 4) is cut into as many K slices as keep every item in one round over the SMs, except a
    small one (8 MB of weights, up to 32 rows), which the streaming kernel does faster; the rest
    streams."""
    tiles = -(-N // 128)
    if tiles >= SM_COUNT // 2:
        return M > 12, 1
    if mode == 4:
        if M <= 32 and N * K <= 4 * 1024 * 1024:
            return False, 1
        k_blocks = -(-K // 64)
        return True, max(1, min(k_blocks, 64, SM_COUNT // tiles))
    return False, 1


def few_takes(M: int, N: int, K: int, mode: int) -> bool:
    """Whole products of 13 to 64 rows that were timed on the kernel with the weights as the wide tcgen05 operand against the tile
    kernel first (few_plan goes on from here): its ring holds 200 KB per SM on their way and reads at 6 TB/s. us in a chain of products
    over more weights than L2 holds, in brackets the tile kernel. bfloat16 results: 16384 x 2048 16 rows 12.2 (14.8), 32 rows 13.0 (15.0),
    28672 x 4096 16 rows 39.1 (46.9), 32 rows 40.3 (47.5), 49408 x 4096 32 rows 65.9 (72.3), 64 rows 70.4 (73.4), 128256 x 2048 64 rows
    84.1 (88.9), 9472 x 22000 32 rows 84.1 (103.4). Gated: 16384 x 2048 16 rows 12.4 (15.5), 32 rows 13.5 (15.4), 28672 x 4096 32 rows 41.0
    (48.2), 49408 x 4096 48 rows 70.9 (73.2)."""
    if not 12 < M <= (48 if mode == 3 else 64):
        return False
    tiles = -(-N // 128)
    return mode in (0, 1, 3) and tiles >= (SM_COUNT // 2 if M <= 32 else SM_COUNT) and N * K >= (30e6 if M <= 32 else 200e6)


def few_plan(M: int, N: int, K: int, mode: int, added: bool = False) -> int:
    """K slices (1: whole) on the kernel with the weights as the wide operand, 0 where another kernel is the faster one. Mode 4 may be
    cut; the others never are. `added`: the slices go to a norm, which adds them to the residual stream.

    Narrow products are cut until their items fill the SMs. us in chains of products, in brackets the streaming or the tile kernel:
    6144 x 4096 in three slices 32 rows 10.3 (22.4), 64 rows 11.5 (40.7); 5120 x 3072 9 rows 7.7 (12.2), 48 rows 9.0 (28.2); 4096 x 14336
    in four 32 rows 21.4 (24.2); 2048 x 8192 in nine 12 rows 7.7 (9.8), 64 rows 9.0 (10.3). Whole: 28672 x 4096 gated 12 rows 39.3 (62.1), 64
    rows 44.5 (47.7); 32768 x 4096 12 rows 43.5 (66.1); 8192 x 2048 24 rows 10.1 (13.1), 12 rows 9.8 (9.3); 5120 x 3072 12 rows 12.5
    (12.7), 64 rows 15.0 (31.5). A norm that adds planes takes 2 to 4 us more than one behind a product that was added in place (2048 x
    2048 16 rows 6.6 against 6.0, 64 rows 8.1 against 10.3), so small products of few rows that go to one stream. Up to 8 rows:
    _few_up_to_eight. Whole steps of two layers and a head of 32,768, before this rule / by it: 1B shape 9 sequences 165 / 141, 48 196 / 182, 3B
    shape 12 268 / 190, 48 288 / 246, 8B shape 12 373 / 274, 48 400 / 343."""
    if M > 64 or mode not in (0, 1, 3, 4):
        return 0
    if few_takes(M, N, K, mode):
        return 1
    tiles = -(-N // 128)
    if M <= STREAM_ROWS:
        if not _few_up_to_eight(M, N, K, mode, added):
            return 0
    elif added and M <= 32 and N * K <= 4 * 1024 * 1024:
        return 0
    if mode == 4:
        k_blocks = -(-K // 64)
        per_slice = max(4, -(-k_blocks // max(1, SM_COUNT // tiles)))
        return -(-k_blocks // per_slice)
    if M <= STREAM_ROWS:
        return 1
    return 1 if tiles >= SM_COUNT // 2 or (min(N, K) >= 3072 and tiles >= 64) or (M > 16 and tiles >= 40) else 0


def _few_up_to_eight(M: int, N: int, K: int, mode: int, added: bool) -> bool:
    """Where up to 8 rows leave the streaming kernel, whose CTAs have 16 columns each. us a whole decode step, streamed / here, by what
    the line is about (all before the weights here left L2 first, which took another 2 to 4 % off the steps):

    * more columns than eight such CTAs an SM have (18,944): a second round of them. Gates, four layers, 1 and 8 sequences: hidden 2,048,
      18,432 columns 172 / 180 and 193 / 195, 19,456 196 / 194 and 227 / 214, 28,672 227 / 222 and 249 / 242; hidden 2,560, 18,432 224 / 230 and
      249 / 247, 19,456 260 / 248 and 296 / 269; hidden 1,024, 19,456 144 / 146 and 162 / 158.
    * gates of fewer columns, but two tiles for every second SM: K above 3,072. 17,920 x 3,328 277 / 277 and 301 / 297, 18,432 x 3,584 279 / 278
      and 305 / 297, 18,432 x 4,096 321 / 317 and 353 / 344; 16,384 x 3,072 248 / 252 and 278 / 279. (64 tiles: 4,096 wide, 8 sequences, 326 / 355.)
    * heads, the same line. Two layers, 1, 4 and 8 sequences: 24,576 x 2,560 127 / 124, 133 / 130, 140 / 135; 98,304 x 2,048 151 / 150, 162 / 158,
      170 / 163; 49,152 x 1,024 78 / 77, 86 / 84, 87 / 87. A single sequence of 2,048 of K may lose: 24,576 107 / 107, 32,768 110 / 112 (4 and 8
      sequences 120 / 119, 124 / 122), six layers 251 / 255.
    * whole bfloat16 results (a q|k|v projection of 74 tiles and more): both sides 3,072 and more, four layers of 12,288 x 4,096 343 / 336 and
      389 / 377.
    * slices that a norm adds up: K of 8,192 and more (which the streaming kernel cuts too) or a third CTA an SM, not where each SM has one.
      A product and its norm, 1 and 8 rows: 2,048 x 8,192 9.8 / 11.9 and 10.5 / 12.3; 2,560 x 8,192 15.4 / 12.5 and 16.4 / 13.3, x 6,144 10.3 / 11.3
      and 10.9 / 12.0; 4,096 x 6,144 12.5 / 14.1 and 13.4 / 14.5, x 8,192 17.3 / 17.0 and 19.0 / 17.3, x 14,336 27.7 / 25.4 and 29.2 / 26.3; 5,120 x
      5,120 15.8 / 14.9 and 16.9 / 15.5; 8,192 x 8,192 31.0 / 27.7 and 32.2 / 28.3.
    * slices that decode attention adds up, every CTA for the rows it needs: large products only. Four layers, 1 and 8 sequences: 3,840 x 3,328
      (13 heads to a key head) 270 / 290 and 284 / 305, 4,608 x 3,584 277 / 292 and 293 / 310, two layers of 5,120 x 3,072 157.6 / 159.4 and 171.6 / 172.8;
      6,144 x 4,096 269 / 269 and 300 / 296, 8,192 x 6,144 317 / 317 and 334 / 332."""
    rounds = -(-N // (16 * SM_COUNT))  # CTAs of the streaming kernel to an SM
    if mode == 4:
        if added:
            return rounds > 1 and (K >= 8192 or rounds > 2)
        return min(N, K) >= 3072 and N * K >= 22e6
    return rounds > 8 or (-(-N // 128) >= SM_COUNT // 2 and (K > 3072 if mode == 3 else min(N, K) >= 3072))


def _few(x: torch.Tensor, weight: torch.Tensor, mode: int, lib, added: bool = False) -> int:
    """few_plan where the kernel takes the product at all."""
    M, K = x.shape
    N = weight.shape[0]
    if (M > 64 or force_tiled or force_stream or stream_shape is not None or umma_width is not None or x.data_ptr() % 16
            or weight.data_ptr() % 16 or (mode == 3 and N % 16)):
        return 0
    slices = few_plan(M, N, K, mode, added)
    return slices if slices and lib.lrm_gemm_bf16_few_supports(M, N, K) else 0


def gemm_bf16_few_slices(x: torch.Tensor, weight: torch.Tensor, added: bool = False) -> Optional[torch.Tensor]:
    """x . weight^T as planes over K slices from that kernel, or None where it is not to be cut there."""
    slices = _few(x, weight, 4, library.load(), added)
    if slices <= 1:
        return None
    out = torch.empty((slices, x.shape[0], weight.shape[0]), dtype=torch.float32, device=x.device)
    gemm_bf16_few(x, weight, out, 4, slices)
    return out


def gemm_bf16_cut(x: torch.Tensor, weight: torch.Tensor) -> Optional[torch.Tensor]:
    """x . weight^T as planes over K slices that the caller adds up at once, or None where the whole product is the better one."""
    M, K = x.shape
    N = weight.shape[0]
    if M > 64:
        if no_wide or umma_width is not None or N % 2 or pair_room() == 0 or not cut_plan(M, N, K, pair_room()):
            return None
        return gemm_bf16_slices(x, weight)
    return gemm_bf16_few_slices(x, weight) if cut_plan(M, N, K, 0) else None


def _held_rows(x: torch.Tensor) -> int:
    """Rows of x, beyond its own, that its storage holds, up to 32 (they may be named in a tensor map)."""
    M, K = x.shape
    held = (x.untyped_storage().nbytes() // x.element_size() - x.storage_offset()) // K
    return min(max(M, 32), max(M, held))


def gemm_bf16_few(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, mode: int, slices: int = 1, rows: int = 0) -> None:
    """gemm_bf16 (modes 0, 1, 3), or K slices as planes (mode 4), for up to 64 rows on the kernel with the weights as the wide operand."""
    M, K = x.shape
    lib = library.load()
    mark_status_dirty()
    _done(lib.lrm_gemm_bf16_few(_ptr(x), _ptr(weight), _ptr(out), M, _held_rows(x), weight.shape[0], K, mode, slices, rows,
                                _ptr(_status_word(x.device)), _stream()), "gemm_bf16_few")


def _fast_kernels(x: torch.Tensor, weight: torch.Tensor, lib):
    M, K = x.shape
    N = weight.shape[0]
    aligned = x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0
    fast = not force_tiled and aligned
    return (fast and bool(lib.lrm_gemm_bf16_stream_supports(M, N, K)),
            fast and bool(lib.lrm_gemm_bf16_umma_supports(M, N, K)))


def _sliced_plan(M: int, N: int, K: int):
    """(tile, K slices) for a product of a few hundred rows that goes into the residual stream as
    planes: 128 x 128 or 128 x 256 tiles, K cut until the items fill the SMs once (no slice shorter
    than 256), whichever is estimated faster, or (0, 1) where the uncut product added in place is.
    Measured per 64 of K and item: 0.30 us with 128 x 128 tiles (0.26 where their operands come from
    L2), 0.35 us with 128 x 256 (twice the work), more where few row tiles share a W tile that comes from HBM; a plane more costs its write
    and the norm's read of it, and the norm adds planes eight at a time. Whole prompt steps of the
    1B shape, this rule against 128 x 128 tiles only: 768 tokens 2.46 against 2.69 ms, 1,024 tokens
    2.92 against 3.03, 128 tokens 1.39 against 1.41, 256 and 512 tokens unchanged."""
    k_blocks = -(-K // 64)
    best, whole = None, None
    row_tiles = -(-M // 128)
    for tile, (columns, per_block) in enumerate(((128, 0.30), (256, 0.35))):
        # with few row tiles a W tile is fetched from HBM for almost every item: 44 GB/s per SM
        per_block = max(per_block, columns * 128 / 44e3 / row_tiles)
        tiles = row_tiles * -(-N // columns)
        uncut = -(-tiles // SM_COUNT) * k_blocks * per_block       # added in place, no planes
        whole = uncut if whole is None else min(whole, uncut)
        fill = max(1, min(k_blocks // 4, SM_COUNT // tiles))
        for splits in {fill, min(fill, 8)}:                        # the norm adds planes eight at a time
            per_slice = -(-k_blocks // splits)
            planes = -(-k_blocks // per_slice)
            rounds = -(-tiles * planes // SM_COUNT)
            cost = (rounds * per_slice * per_block + planes * (2.0 * M * N * 4 / 3.5e6)
                    + 2.0 * (-(-planes // 8) - 1))
            if planes > 1 and (best is None or cost < best[0]):
                best = (cost, tile, splits)
    if best is None or best[0] >= whole:
        return 0, 1                                               # not worth cutting
    return best[1], best[2]


def gemm_bf16_slices(x: torch.Tensor, weight: torch.Tensor) -> Optional[torch.Tensor]:
    """x . weight^T as float32 partial products over K slices, [slices, M, N], whose sum in plane
    order is the product; None when this shape is not worth cutting (the caller then adds the
    whole product in place). For products that go into the residual stream."""
    M, K = x.shape
    N = weight.shape[0]
    lib = library.load()
    planes = gemm_bf16_few_slices(x, weight, added=True)
    if planes is not None:
        return planes
    stream_ok, umma_ok = _fast_kernels(x, weight, lib)
    if not stream_ok:
        if not umma_ok or M <= 64:
            return None
        # A short prompt (a few hundred rows): few tiles and a long K leave most SMs idle (the 2048 x
        # 8192 product of a 128-token prompt: 16 CTAs, 42 us), so K is cut until the items fill the
        # SMs once, no slice shorter than 256 (the same product in 9 slices: 12 us).
        wide = _wide(x, weight, 2, umma_ok)
        if wide is not None:
            if wide[1] == 1:
                return None
            out = torch.empty((wide[1], M, N), dtype=torch.float32, device=x.device)
            gemm_bf16_wide(x, weight, out, 4, *wide)
            return out
        tile, splits = _sliced_plan(M, N, K)
        planes = lib.lrm_gemm_bf16_umma_slices(K, splits) if splits > 1 else 1
        if planes <= 1:
            return None
        out = torch.empty((planes, M, N), dtype=torch.float32, device=x.device)
        mark_status_dirty()
        _done(lib.lrm_gemm_bf16_umma_rows(_ptr(x), _ptr(weight), _ptr(out), M, M, N, K, 4, tile, splits,
                                          _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma")
        return out
    use_umma, splits = False, 1
    if umma_ok and M > STREAM_ROWS and not force_stream:
        use_umma, splits = _few_rows_plan(M, N, K, 4)
    if use_umma:
        planes = lib.lrm_gemm_bf16_umma_slices(K, splits)
        if planes <= 1:
            return None
        out = torch.empty((planes, M, N), dtype=torch.float32, device=x.device)
        mark_status_dirty()
        held = (x.untyped_storage().nbytes() // x.element_size() - x.storage_offset()) // K
        _done(lib.lrm_gemm_bf16_umma_rows(_ptr(x), _ptr(weight), _ptr(out), M, min(max(M, 32), max(M, held)), N, K,
                                          4, 0 if umma_width is None else tile_choice(M, N, K, 4), splits,
                                          _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma")
        return out
    warps, wanted = stream_shape if stream_shape is not None else (0, 0)
    planes = lib.lrm_gemm_bf16_stream_slices(M, N, K, wanted)
    if planes <= 1:
        return None
    out = torch.empty((planes, M, N), dtype=torch.float32, device=x.device)
    _done(lib.lrm_gemm_bf16_stream_shaped(_ptr(x), _ptr(weight), _ptr(out), M, N, K, 4, warps, wanted, _stream()),
          "gemm_bf16_stream")
    return out


def qkv_apart(M: int, N: int, K: int) -> bool:
    """Whether a prompt's q|k|v projection goes to the tiles with the weights as the wide operand and the rotation and the stores to a
    launch of their own, instead of tiles with the activations as the wide operand that rotate and store in their epilogue (gemm_bf16_qkv;
    the same bits): rows that leave those tiles half empty, and matrices whose gain is more than the host's time for the launch where a
    length comes for the first time and is not replayed (3072 x 2048, four layers, 66 and 256 tokens: in one 860 and 890 us, apart 920 and
    950; replayed 306 and 337, apart 294 and 319; 560 tokens 430 either way). us in
    chains of weights from memory, apart and in one: 6144 x 4096 65 rows 18 and 25, 320 23 and 26, 529 28 and 31, 700 33 and 32; 5120 x 3072 65
    rows 15 and 20, 529 23 and 27, 700 28 and 27; 10240 x 8192 192 rows 44 and 51, 256 53 and 51; 12288 x 4096 128 rows 29 and 32, 320 39 and 37;
    3072 x 2048, below the line, 65 rows 12 and 15, 400 14 and 16."""
    return (not no_wide and umma_width is None and 64 < M <= (560 if N * K <= 32e6 else 200) and N * K >= 12e6
            and pair_room() > 0 and wide_plan(M, N, K, 0, pair_room()) is not None)


def gemm_bf16_qkv(x: torch.Tensor, weight: torch.Tensor, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
                  kv, dest_rows: Optional[torch.Tensor], table: Optional[torch.Tensor]) -> bool:
    """A prompt's fused q|k|v projection with rotation and stores in the product's epilogue:
    q [T, Hq, d], k, v [T, Hk, d] packed, and k, v into the paged cache view `kv` at `dest_rows`
    (both None: no cache). `table`: float32 [T, d/2, 2] (cos, sin), or None for no rotation.
    False (nothing launched) where only the separate kernels take the shape."""
    M, K = x.shape
    N = weight.shape[0]
    T, Hq, d = q.shape
    Hk = k.shape[1]
    lib = library.load()
    _, umma_ok = _fast_kernels(x, weight, lib)
    if not umma_ok or no_fused_rope or M <= 64 or d not in (64, 128) or N != (Hq + 2 * Hk) * d:
        return False
    tile = tile_choice(M, N, K, 0, pair_room(), multiple_of=d)
    pages = (_ptr(kv.k), _ptr(kv.v), _ptr(dest_rows), kv.page_size) if kv is not None else (None, None, None, 1)
    mark_status_dirty()
    if tile == PAIR:
        _done(lib.lrm_gemm_bf16_umma_pair_qkv(_ptr(x), _ptr(weight), M, N, K, _ptr(q), _ptr(k), _ptr(v), pages[0],
                                              pages[1], pages[2], _ptr(table), Hq, Hk, d, pages[3],
                                              _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma_pair_qkv")
    else:
        _done(lib.lrm_gemm_bf16_umma_qkv(_ptr(x), _ptr(weight), M, N, K, tile, _ptr(q), _ptr(k), _ptr(v), pages[0],
                                         pages[1], pages[2], _ptr(table), Hq, Hk, d, pages[3],
                                         _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma_qkv")
    return True


no_fused_rope = False  # tests: keep rotation and stores in their own launch
no_fused_gate = False  # tests: keep the sorted experts' gate in its own launch


def gemm_bf16(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, mode: int) -> None:
    """out (mode 0 bf16 store, 1 f32 store, 2 f32 add in place, 3 silu gate) = x . weight^T."""
    M, K = x.shape
    N = weight.shape[0]
    lib = library.load()
    if M <= 64 and _few(x, weight, mode, lib):
        gemm_bf16_few(x, weight, out, mode)
        return
    stream_ok, umma_ok = _fast_kernels(x, weight, lib)
    if M > 64 and mode <= 3 and out.data_ptr() % 4 == 0:
        wide = _wide(x, weight, 1 if mode == 2 else mode, umma_ok)  # whole: out takes no planes
        if wide is not None:
            gemm_bf16_wide(x, weight, out, mode, wide[0])
            return
    tile, splits = tile_choice(M, N, K, mode, pair_room() if umma_ok and M > 64 else 0), 1
    if stream_ok and umma_ok and M > STREAM_ROWS and not force_stream:
        use_umma, splits = _few_rows_plan(M, N, K, mode)
        stream_ok = not use_umma
        tile = 0 if umma_width is None else tile
    if stream_ok:
        warps = stream_shape[0] if stream_shape is not None else 0
        _done(lib.lrm_gemm_bf16_stream_shaped(_ptr(x), _ptr(weight), _ptr(out), M, N, K, mode, warps, 0,
                                              _stream()), "gemm_bf16_stream")
        return
    if umma_ok and tile == PAIR:
        mark_status_dirty()
        _done(lib.lrm_gemm_bf16_umma_pair(_ptr(x), _ptr(weight), _ptr(out), M, N, K, mode,
                                          _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma_pair")
        return
    if umma_ok:
        mark_status_dirty()
        # rows of x that its storage holds beyond M may be named in the tensor map (see the kernel)
        held = (x.untyped_storage().nbytes() // x.element_size() - x.storage_offset()) // K
        _done(lib.lrm_gemm_bf16_umma_rows(_ptr(x), _ptr(weight), _ptr(out), M, min(max(M, 32), max(M, held)), N, K,
                                          mode, tile, splits, _ptr(_status_word(x.device)), _stream()),
              "gemm_bf16_umma")
        return
    _done(lib.lrm_gemm_bf16_mma(_ptr(x), _ptr(weight), _ptr(out), M, N, K, mode, _stream()),
          "gemm_bf16_mma")


def f32_takes_umma(N: int, K: int) -> bool:
    """Whether a float32 product goes to the tensor cores in three-part splits (csrc/gemm_f32_umma.cu) or to the FMA kernels
    (csrc/gemm_f32.cu). A matter of the matrix alone, so that a row gives the same bits however many there are. us for 1, 32 and 333
    rows, in brackets the FMA kernels: 1024 x 1024 9.9 (12.7), 11.1 (28.7), 18.2 (40.0); 512 x 2048 9.9 (24.2), 11.6 (56.2), 21.0
    (76.2); 2048 x 512, below the line, 9.2 (6.9), 10.6 (17.4), 18.9 (33.2). Of larger matrices a single row of 128256 x 2048 alone is slower (196 against 175; 4 rows 197 against 240). Rows on 32 bytes (K a multiple of 8), as the parts' copies want them."""
    return K % 8 == 0 and K >= 1024 and N >= 512


def gemm_f32(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, mode: int, rows: int, group_cols: int = 0) -> None:
    """float32 out [rows, N] (mode 0: =, 1: +=) x . weight^T. group_cols > 0: columns i * group_cols .. belong to the input that begins
    i * rows rows into x. The kernel follows from the matrix and the addresses alone, never from `rows`."""
    N, K = weight.shape
    lib = library.load()
    if (f32_takes_umma(N, K) and not force_tiled and group_cols % 128 == 0 and x.data_ptr() % 16 == 0
            and weight.data_ptr() % 16 == 0):
        mark_status_dirty()
        scratch = lib.lrm_gemm_f32_umma_scratch(rows, x.numel() // K, K)
        parts = torch.empty(scratch, dtype=torch.uint8, device=x.device) if scratch else None
        _done(lib.lrm_gemm_f32_umma(_ptr(x), _ptr(weight), _ptr(out), rows, N, K, mode, group_cols, rows, _ptr(parts),
                                    _ptr(_status_word(x.device)), _stream()), "gemm_f32_umma", launches=2 if scratch else 1)
        return
    if group_cols:
        _done(lib.lrm_gemm_f32_grouped(_ptr(x), _ptr(weight), _ptr(out), rows, N, K, mode, group_cols, rows, _stream()),
              "gemm_f32_grouped")
    else:
        _done(lib.lrm_gemm_f32(_ptr(x), _ptr(weight), _ptr(out), rows, N, K, mode, _stream()), "gemm_f32")


def gemm_bf16_split(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, gated: torch.Tensor) -> None:
    """Two products with one input: out (float32 [M, split]) = x . weight[:split]^T, and the SiLU gate of the gate
    and up rows behind it into the first columns of `gated` (bfloat16 [M, W]). One launch of the kernels of
    gemm_bf16; two where only the warp-level kernel takes the shape."""
    M, K = x.shape
    N, split, pitch = weight.shape[0], out.shape[1], gated.shape[1]
    lib = library.load()
    stream_ok, umma_ok = _fast_kernels(x, weight, lib)
    if stream_ok and umma_ok and M > STREAM_ROWS and not force_stream:
        stream_ok = not _few_rows_plan(M, N, K, 6)[0]
    where = (_ptr(x), _ptr(weight), _ptr(out), split, _ptr(gated), ctypes.c_longlong(pitch), M)
    if stream_ok:
        _done(lib.lrm_gemm_bf16_stream_split(*where, N, K, _stream()), "gemm_bf16_stream_split")
        return
    if umma_ok and pitch % 8 == 0:
        tile = tile_choice(M, N, K, 1, pair_room() if M > 64 else 0)
        mark_status_dirty()
        if tile == PAIR:
            _done(lib.lrm_gemm_bf16_umma_pair_split(*where, N, K, _ptr(_status_word(x.device)), _stream()),
                  "gemm_bf16_umma_pair_split")
            return
        held = (x.untyped_storage().nbytes() // x.element_size() - x.storage_offset()) // K
        _done(lib.lrm_gemm_bf16_umma_split(*where, min(max(M, 32), max(M, held)), N, K, tile, _ptr(_status_word(x.device)),
                                           _stream()), "gemm_bf16_umma_split")
        return
    _done(lib.lrm_gemm_bf16_mma(_ptr(x), _ptr(weight), _ptr(out), M, split, K, 1, _stream()), "gemm_bf16_mma")
    _done(lib.lrm_gemm_bf16_mma_gate(_ptr(x), _ptr(weight[split:]), _ptr(gated), ctypes.c_longlong(pitch), M, N - split, K,
                                     _stream()), "gemm_bf16_mma_gate")


def gemm_bf16_grouped(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, group_cols: int) -> None:
    """float32 out [T, N] from the inputs x [G, T, K] and one stacked weight [N, K]: columns i * group_cols
    .. of out belong to x[i]. The kernels of gemm_bf16 with a row offset into x per column tile."""
    G, T, K = x.shape
    N = weight.shape[0]
    lib = library.load()
    aligned = not force_tiled and x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0
    stream_ok = aligned and bool(lib.lrm_gemm_bf16_stream_supports(T, N, K))
    umma_ok = aligned and bool(lib.lrm_gemm_bf16_umma_supports(T, N, K))
    if stream_ok and umma_ok and T > STREAM_ROWS and not force_stream:
        stream_ok = not _few_rows_plan(T, N, K, 1)[0]
    if stream_ok:
        _done(lib.lrm_gemm_bf16_stream_grouped(_ptr(x), _ptr(weight), _ptr(out), T, N, K, 1, group_cols, T, _stream()),
              "gemm_bf16_stream_grouped")
        return
    if umma_ok:
        tile = tile_choice(T, N, K, 1, pair_room() if T > 64 else 0)
        width = {0: 128, 1: 256, 2: 256, 3: 192, PAIR: 256}[tile]
        if group_cols % width:
            tile = 1 if group_cols % 256 == 0 else 0
        mark_status_dirty()
        if tile == PAIR:
            _done(lib.lrm_gemm_bf16_umma_pair_grouped(_ptr(x), _ptr(weight), _ptr(out), T, G * T, N, K, 1, group_cols, T,
                                                      _ptr(_status_word(x.device)), _stream()),
                  "gemm_bf16_umma_pair_grouped")
        else:
            _done(lib.lrm_gemm_bf16_umma_grouped(_ptr(x), _ptr(weight), _ptr(out), T, G * T, N, K, 1, tile, group_cols, T,
                                                 _ptr(_status_word(x.device)), _stream()), "gemm_bf16_umma_grouped")
        return
    _done(lib.lrm_gemm_bf16_mma_grouped(_ptr(x), _ptr(weight), _ptr(out), T, N, K, 1, group_cols, T, _stream()),
          "gemm_bf16_mma_grouped")
